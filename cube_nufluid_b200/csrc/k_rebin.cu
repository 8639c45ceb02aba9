/*
 * k_rebin.cu -- update_x: drift, re-bin by counting sort, re-encode
 * (update_particle.f90:13-259).
 *
 * The reference drifts every particle of a tile plus its ncb-cell buffer,
 * counts the new cells, builds the spine, scatters in its loop order
 * (layer, k, j, i, l) with nlayer = 2*ceiling(dt_mid*vz_max/ncell)+1, and
 * keeps the particles that land in the tile.  Inside a new cell the particles
 * therefore sit in that loop order, and the cell's new mean velocity is an
 * FP32 running sum in the same order.  The GPU reproduces both exactly:
 *
 *   count   : per particle, target cell (computed in the coordinates of the
 *             target tile, as the reference does) and a 32-bit order key
 *             ((layer*nte + k)*nte + j)*nte + i of the source cell in those
 *             coordinates; count per target cell
 *   scan    : cell starts
 *   place   : slot = start + atomic cursor (arbitrary order inside the cell)
 *   cells   : per group of target cells, one thread per entry: its rank among the
 *             cell's (key, source index) pairs -- the reference order -- places its
 *             velocity in shared memory; the FP32 velocity sums run in that order, one
 *             thread per cell and component, with the division by (n + weight_v); then
 *             every entry is re-encoded against the new mean, moved and written
 *             to its slot with its PID.  Cells with more than 32 particles go to a
 *             warp sorter (one warp per cell, many cells per SM, so the serial sums of
 *             different cells overlap), those beyond 256 to a block-wide sorter in
 *             shared memory, those beyond 4096 to one in a global scratch grown on
 *             demand; emit then writes their entries
 *   stats   : per cell |vfield|^2, summed by the fixed tree
 * Positions move by nint(dt_mid*v/(x_resolution*ncell)) with the integer
 * wrap of the 1- or 2-byte store (update_particle.f90:117).
 */
#include "cube_internal.cuh"

#include <algorithm>
#include <cmath>

namespace {

constexpr int RCELLS = 64;  // cube_cell_item assumes 64-cell groups
constexpr int PMAX = 4096;     // particles per work item of the count and emit passes
constexpr int SMALL = 32;
static_assert(SMALL * RCELLS <= PMAX, "a group of uncrowded cells is one work item");
constexpr int WARP_MAX = 256;  // warp sorter: keys + 3 velocity columns, 8 KB per warp
constexpr int WARP_WARPS = 8;
constexpr int BIG_MAX = 4096;

struct RebinArgs {
  const void* xp; const void* vp; const int32_t* pid;
  const int64_t* cell_start; const float* vfield;
  void* xp2; void* vp2; int32_t* pid2;
  int32_t* cnt2; int64_t* start2; float* vfield2;
  int32_t* tcell; uint32_t* tkey; int32_t* perm; uint32_t* pkey; int32_t* cursor;
  int32_t* big_list; int32_t* slot_cell;  // new cell of each slot
  const int64_t* items; int64_t items_max;
  const double* dec; int half_nvbin;  // tan(code)/coef per code (cube_vdec_table)
  cube_codec codec; double coef; VencTab tab;
  double inv_ncell, inv_xstep;  // 1/ncell and 1/(x_resolution*ncell), exact powers of two
  int64_t cap, ncells;
  int nc, nt, nnt, ncb, nte, ncell, nlayer, use_pid;
  FastDiv dnt, dnt3, dnnt, dnte, dnlayer;  // nt, nt^3, nnt; nte and nlayer over keys and source rows
  float dt_mid;
  DevScal* dscal;
};

// cube_cell_of with the division by nt as a multiply
__device__ __forceinline__ int64_t cell_of(const RebinArgs& A, int gx, int gy, int gz) {
  const int nt = A.nt, tx = (int)((uint32_t)gx / A.dnt), ty = (int)((uint32_t)gy / A.dnt), tz = (int)((uint32_t)gz / A.dnt);
  const int lx = gx - tx * nt, ly = gy - ty * nt, lz = gz - tz * nt;
  return ((((int64_t)tz * A.nnt + ty) * A.nnt + tx) * nt + lz) * (int64_t)nt * nt + (int64_t)ly * nt + lx;
}

__device__ __forceinline__ int floordiv(int a, int b) { return (a >= 0) ? a / b : -((-a + b - 1) / b); }

template <int ZX, int ZV>
__device__ __forceinline__ double decode_v(const RebinArgs& A, int64_t ip, int d) {
  typedef typename CodeT<ZV>::T TV;
  const TV* vp = reinterpret_cast<const TV*>(A.vp);
  const int code = (int)vp[(size_t)d * A.cap + ip];
  return __ldg(&A.dec[code + A.half_nvbin]);
}

// Work items of the count and emit passes (and of the kick): a run of at most
// RCELLS cells and a particle range inside it of at most PMAX particles.  Item
// g < ngroups is the 64-cell group g (all of it when it holds at most PMAX
// particles); a crowded group is cut greedily into runs of whole cells, a cell
// beyond PMAX particles into ranges of PMAX, and the items after its first are
// appended after the groups.  A group of cnt > PMAX particles makes at most
// 4 cnt/PMAX items.
__device__ __forceinline__ void put_item(int64_t* items, int64_t items_max, int64_t ngroups, DevScal* dscal, int64_t g,
                                         bool& first, int64_t c0, int64_t ncl, int64_t p0, int64_t p1) {
  int64_t idx = g;
  if (!first) {
    idx = ngroups + (int64_t)atomicAdd(&dscal->n_items, 1ull);
    if (idx >= items_max) {
      cube_dev_error(dscal, CUBE_ERR_CAPACITY, (int)(g & 0x7fffffff));
      return;
    }
  }
  first = false;
  int64_t* it = items + 4 * idx;
  it[0] = c0; it[1] = ncl; it[2] = p0; it[3] = p1;
}

__global__ void k_cell_items(const int64_t* __restrict__ cs, int64_t ncells, int64_t* __restrict__ items,
                             int64_t items_max, DevScal* dscal) {
  const int64_t ngroups = (ncells + RCELLS - 1) / RCELLS;
  const int64_t g = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (g >= ngroups) return;
  const int64_t c0 = g * RCELLS;
  const int64_t ncl = min((int64_t)RCELLS, ncells - c0);
  bool first = true;
  if (cs[c0 + ncl] - cs[c0] <= PMAX) {
    put_item(items, items_max, ngroups, dscal, g, first, c0, ncl, cs[c0], cs[c0 + ncl]);
    return;
  }
  int64_t ic = c0;  // first cell of the open run
  for (int64_t c = c0; c < c0 + ncl; ++c) {
    const int64_t a = cs[c], e = cs[c + 1];
    if (e - a > PMAX) {
      if (c > ic) put_item(items, items_max, ngroups, dscal, g, first, ic, c - ic, cs[ic], a);
      for (int64_t q = a; q < e; q += PMAX)
        put_item(items, items_max, ngroups, dscal, g, first, c, 1, q, min(q + PMAX, e));
      ic = c + 1;
    } else if (e - cs[ic] > PMAX) {  // cell c does not fit the open run (c > ic here)
      put_item(items, items_max, ngroups, dscal, g, first, ic, c - ic, cs[ic], a);
      ic = c;
    }
  }
  if (c0 + ncl > ic) put_item(items, items_max, ngroups, dscal, g, first, ic, c0 + ncl - ic, cs[ic], cs[c0 + ncl]);
}

// item of this block, or false past the last
__device__ __forceinline__ bool get_item(const RebinArgs& A, int64_t& c0, int& ncl, int64_t& p0, int64_t& p1) {
  return cube_cell_item(A.items, A.ncells, A.items_max, A.dscal, A.cell_start, (int64_t)blockIdx.x, c0, ncl, p0, p1);
}

template <int ZX, int ZV>
__global__ void __launch_bounds__(256) k_rebin_count(RebinArgs A) {
  typedef typename CodeT<ZX>::T TX;
  const TX* xp = reinterpret_cast<const TX*>(A.xp);
  __shared__ int64_t cs[RCELLS + 1];
  __shared__ int cl[RCELLS][3], ctt[RCELLS][3];  // per cell: local coords, tile coords
  int64_t c0, p0, p1;
  int ncl;
  if (!get_item(A, c0, ncl, p0, p1)) return;
  const int nt = A.nt, nnt = A.nnt, ncb = A.ncb, nte = A.nte;
  for (int i = threadIdx.x; i <= ncl; i += blockDim.x) cs[i] = A.cell_start[c0 + i];
  for (int i = threadIdx.x; i < ncl; i += blockDim.x) {
    int tb[3];
    cube_cell_coords(c0 + i, nt, nnt, cl[i], tb);
    ctt[i][0] = tb[0] / nt;
    ctt[i][1] = tb[1] / nt;
    ctt[i][2] = tb[2] / nt;
  }
  __syncthreads();
  typedef typename CodeT<ZV>::T TV;
  const TV* vp = reinterpret_cast<const TV*>(A.vp);
  // two particles per thread, their code and cell-mean reads issued together
  for (int64_t ib = p0 + threadIdx.x; ib < p1; ib += 2 * blockDim.x) {
    int lov[2];
    int xcv[2][3];
    double vv[2][3];
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int64_t q = ib + u * (int64_t)blockDim.x < p1 ? ib + u * (int64_t)blockDim.x : ib;
      int lo = 0, hi = ncl - 1;
      while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (cs[mid] <= q) lo = mid; else hi = mid - 1;
      }
      lov[u] = lo;
      const int64_t c = c0 + lo;
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        xcv[u][d] = (int32_t)xp[(size_t)d * A.cap + q];
        vv[u][d] = cube_dadd(__ldg(&A.dec[(int)vp[(size_t)d * A.cap + q] + A.half_nvbin]),
                             (double)__ldg(&A.vfield[(size_t)d * A.ncells + c]));
      }
    }
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int64_t ip = ib + u * (int64_t)blockDim.x;
      if (ip >= p1) continue;
      const int lo = lov[u];
      const int l[3] = {cl[lo][0], cl[lo][1], cl[lo][2]};
      const int t[3] = {ctt[lo][0], ctt[lo][1], ctt[lo][2]};
      int tg[3], src[3];
      bool bad = false;
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        const double fr = cube_xfrac(xcv[u][d], ZX);
        const double v = vv[u][d];
        // /ncell: ncell = 4 (cube_create), and a quotient by a power of two is the product by
        // its reciprocal, bit for bit
        const double dx = cube_dmul(cube_dmul((double)A.dt_mid, v), A.inv_ncell);
        // ig = ceiling(xq + deltax), xq = (i-1) + frac in the coordinates of the tile that keeps it
        int ig = (int)ceil(cube_dadd(cube_dadd((double)l[d], fr), dx));
        int ls = l[d], tt = t[d];
        if (ig < 1 || ig > nt) {
          const int sh = floordiv(ig - 1, nt);
          ls = l[d] - sh * nt;
          tt = ((t[d] + sh) % nnt + nnt) % nnt;
          const int ig2 = (int)ceil(cube_dadd(cube_dadd((double)ls, fr), dx));
          if (ig2 >= 1 && ig2 <= nt) ig = ig2;
          else { ig = ig - sh * nt; atomicAdd(&A.dscal->moved_far, 1ull); }
        }
        if (ls + 1 < 1 - ncb || ls + 1 > nt + ncb) bad = true;
        tg[d] = tt * nt + ig - 1;
        src[d] = ls + ncb;  // 0-based index in the target tile's extended range
      }
      if (bad) {
        cube_dev_error(A.dscal, CUBE_ERR_MOVE, (int)(ip & 0x7fffffff));
        src[0] = min(max(src[0], 0), nte - 1);
        src[1] = min(max(src[1], 0), nte - 1);
        src[2] = min(max(src[2], 0), nte - 1);
      }
      const int64_t tc = cell_of(A, tg[0], tg[1], tg[2]);
      const uint32_t layer = (uint32_t)src[2] - (uint32_t)src[2] / A.dnlayer * A.nlayer;
      const uint32_t key = ((layer * nte + src[2]) * nte + src[1]) * nte + src[0];
      A.tcell[ip] = (int32_t)tc;
      A.tkey[ip] = key;
      atomicAdd(&A.cnt2[tc], 1);
    }
  }
}

__global__ void k_rebin_place(RebinArgs A, int64_t np) {
  for (int64_t ip = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; ip < np; ip += (int64_t)gridDim.x * blockDim.x) {
    const int32_t tc = A.tcell[ip];
    const int64_t slot = A.start2[tc] + atomicAdd(&A.cursor[tc], 1);
    A.perm[slot] = (int32_t)ip;
    A.pkey[slot] = A.tkey[ip];
  }
}

// source cell of an entry from its key and the target cell's tile
__device__ __forceinline__ int64_t src_cell(const RebinArgs& A, uint32_t key, const int tt[3]) {
  const uint32_t nte = A.nte;
  const uint32_t k1 = key / A.dnte, k2 = k1 / A.dnte;
  const int i = (int)(key - k1 * nte), j = (int)(k1 - k2 * nte), k = (int)(k2 - k2 / A.dnte * nte);
  const int gx = cube_wrap(tt[0] * A.nt + i - A.ncb, A.nc);
  const int gy = cube_wrap(tt[1] * A.nt + j - A.ncb, A.nc);
  const int gz = cube_wrap(tt[2] * A.nt + k - A.ncb, A.nc);
  return cell_of(A, gx, gy, gz);
}

__device__ __forceinline__ void cell_tile(const RebinArgs& A, int64_t c, int tt[3]) {
  const uint32_t tile = (uint32_t)c / A.dnt3;
  const uint32_t q = tile / A.dnnt, r = q / A.dnnt;
  tt[0] = (int)(tile - q * A.nnt);
  tt[1] = (int)(q - r * A.nnt);
  tt[2] = (int)r;
}

// one particle to its slot of the new layout: moved by nint(dt_mid*v/(x_resolution*
// ncell)) (a power of two: the product by its reciprocal, bit for bit), re-encoded
// against the new cell mean, its PID copied
template <int ZX, int ZV>
__device__ __forceinline__ void emit_one(const RebinArgs& A, int64_t c, int64_t slot, int64_t ip, const double v[3],
                                         const float vfn[3]) {
  typedef typename CodeT<ZX>::T TX;
  typedef typename CodeT<ZV>::T TV;
  const TX* xp = reinterpret_cast<const TX*>(A.xp);
  TX* xp2 = reinterpret_cast<TX*>(A.xp2);
  TV* vp2 = reinterpret_cast<TV*>(A.vp2);
  int xc[3];
#pragma unroll
  for (int d = 0; d < 3; ++d) xc[d] = (int)xp[(size_t)d * A.cap + ip];
  const int32_t id = A.use_pid ? A.pid[ip] : 0;
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const int64_t mv = cube_nint(cube_dmul(cube_dmul((double)A.dt_mid, v[d]), A.inv_xstep));
    xp2[(size_t)d * A.cap + slot] = (TX)cube_wrap_code((int64_t)xc[d] + (int32_t)mv, ZX);
    vp2[(size_t)d * A.cap + slot] =
        (TV)cube_wrap_code(cube_vencode_step(&A.codec, A.tab, cube_dsub(v[d], (double)vfn[d]), A.coef), ZV);
  }
  if (A.use_pid) A.pid2[slot] = id;
  A.slot_cell[slot] = (int32_t)c;
}

// the decoded velocity of entry (key, ip) of a cell in tile tt
template <int ZV>
__device__ __forceinline__ void entry_velocity(const RebinArgs& A, uint32_t key, int64_t ip, const int tt[3],
                                               double v[3]) {
  typedef typename CodeT<ZV>::T TV;
  const TV* vp = reinterpret_cast<const TV*>(A.vp);
  int code[3];
#pragma unroll
  for (int d = 0; d < 3; ++d) code[d] = (int)vp[(size_t)d * A.cap + ip];
  const int64_t sc = src_cell(A, key, tt);
#pragma unroll
  for (int d = 0; d < 3; ++d)
    v[d] = cube_dadd(__ldg(&A.dec[code[d] + A.half_nvbin]), (double)__ldg(&A.vfield[(size_t)d * A.ncells + sc]));
}

// F1: GCELLS target cells per CTA, up to GCAP of their entries at a time (whole cells).
// Crowded cells are listed for the sorter of their size: up to WARP_MAX entries at
// the front of big_list (k_rebin_warp), up to BIG_MAX at its back (k_rebin_big),
// beyond that in cursor, which is free after the place pass (k_rebin_huge).
// One thread per entry throughout but for the sums, so the dependent reads (entry,
// codes, decode table, cell means) of many entries are in flight; the passes that this
// replaces (a thread per cell sorting and summing its entries, 3.9 ms at 512^3
// particles, and an emit pass over the old order that decoded them again, 3.6 ms)
// waited on them one entry at a time with 23 of 32 lanes.  This pass: 4.7 ms.
constexpr int GCELLS = 32;
constexpr int GCAP = 384;
constexpr int GTHREADS = 128;
static_assert(SMALL <= GCAP, "a cell's entries fit one batch");

template <int ZX, int ZV>
__global__ void __launch_bounds__(GTHREADS) k_rebin_cells(RebinArgs A) {
  __shared__ unsigned long long ek[GCAP];  // (key, source) of the batch's entries, in slot order
  __shared__ double sv[3][GCAP];           // velocities in the reference order
  __shared__ int32_t sip[GCAP];            // sources in the reference order
  __shared__ uint8_t ec[GCAP];             // cell of each entry
  __shared__ int64_t cs[GCELLS];
  __shared__ int cn[GCELLS], pre[GCELLS + 1], ctt[GCELLS][3];
  __shared__ float vfn[3][GCELLS];
  const int64_t c0 = (int64_t)blockIdx.x * GCELLS;
  const int ncl = (int)min((int64_t)GCELLS, A.ncells - c0);
  const int tid = threadIdx.x, lane = tid & 31;
  if (tid < 32) {
    int n = 0;
    if (lane < ncl) {
      const int64_t c = c0 + lane;
      n = A.cnt2[c];
      cs[lane] = A.start2[c];
      cell_tile(A, c, ctt[lane]);
      cn[lane] = n;
      if (n > SMALL) {
        if (n <= WARP_MAX) {
          A.big_list[atomicAdd(&A.dscal->n_big, 1ull)] = (int32_t)c;
        } else if (n <= BIG_MAX) {
          A.big_list[A.ncells - 1 - (int64_t)atomicAdd(&A.dscal->n_mid, 1ull)] = (int32_t)c;
        } else {
          A.cursor[atomicAdd(&A.dscal->n_huge, 1ull)] = (int32_t)c;
          atomicMax(&A.dscal->max_huge, (unsigned long long)n);
        }
        cn[lane] = -1;
        n = 0;
      }
    }
    int inc = n;
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += v;
    }
    pre[lane + 1] = inc;
    if (lane == 0) pre[0] = 0;
  }
  __syncthreads();
  for (int ca = 0; ca < ncl;) {
    const int b0 = pre[ca];
    // as many whole cells as fit the batch (a prefix of the cells from ca on)
    const unsigned fit = __ballot_sync(0xffffffffu, lane >= ca && lane < ncl && pre[lane + 1] - b0 <= GCAP);
    const int w = __popc(fit), tot = pre[ca + w] - b0;
    for (int t = tid; t < tot; t += GTHREADS) {
      int lo = ca, hi = ca + w - 1;  // last cell whose first entry is not beyond t
      while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (pre[mid] - b0 <= t) lo = mid; else hi = mid - 1;
      }
      const int64_t s = cs[lo] + (t + b0 - pre[lo]);
      ek[t] = ((unsigned long long)A.pkey[s] << 32) | (uint32_t)A.perm[s];
      ec[t] = (uint8_t)lo;
    }
    __syncthreads();
    for (int t = tid; t < tot; t += GTHREADS) {
      const int ci = ec[t], k0 = pre[ci] - b0, n = cn[ci];
      const unsigned long long me = ek[t];
      int rank = 0;
      for (int j = 0; j < n; ++j) rank += ek[k0 + j] < me;
      const int32_t ip = (int32_t)(uint32_t)me;
      double v[3];
      entry_velocity<ZV>(A, (uint32_t)(me >> 32), ip, ctt[ci], v);
      sip[k0 + rank] = ip;
#pragma unroll
      for (int d = 0; d < 3; ++d) sv[d][k0 + rank] = v[d];
    }
    __syncthreads();
    // the cells' FP32 sums in that order (update_particle.f90:74,83-85)
    for (int t = tid; t < 3 * w; t += GTHREADS) {
      const int d = t / w, ci = ca + t - d * w, n = cn[ci];
      if (n < 0) continue;
      const int64_t c = c0 + ci;
      const double* x = sv[d] + (pre[ci] - b0);
      float acc = (float)cube_dmul((double)A.vfield[(size_t)d * A.ncells + c], 0.1);
      for (int i = 0; i < n; ++i) acc = (float)cube_dadd((double)acc, x[i]);
      const float m = (float)cube_ddiv((double)acc, cube_dadd((double)n, 0.1));
      vfn[d][ci] = m;
      A.vfield2[(size_t)d * A.ncells + c] = m;
    }
    __syncthreads();
    for (int t = tid; t < tot; t += GTHREADS) {
      const int ci = ec[t];
      const double v[3] = {sv[0][t], sv[1][t], sv[2][t]};
      const float m[3] = {vfn[0][ci], vfn[1][ci], vfn[2][ci]};
      emit_one<ZX, ZV>(A, c0 + ci, cs[ci] + (t + b0 - pre[ci]), sip[t], v, m);
    }
    __syncthreads();
    ca += w;
  }
}

// acc + x[0] + x[1] + ... + x[n-1] left to right, each partial sum rounded to FP32
// through FP64 (the reference's real(4) accumulation of real(8) terms); the loads of
// eight terms are issued ahead of their adds
__device__ __forceinline__ float ordered_sum_lane(float acc, const double* x, int n) {
  int i = 0;
  for (; i + 8 <= n; i += 8) {
    double t[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) t[u] = x[i + u];
#pragma unroll
    for (int u = 0; u < 8; ++u) acc = (float)cube_dadd((double)acc, t[u]);
  }
  for (; i < n; ++i) acc = (float)cube_dadd((double)acc, x[i]);
  return acc;
}

// The same sum by a warp, for the sorters whose time is one cell's; every lane passes and
// returns the same acc.  Above, a term is a chain of convert, FP64 add and convert, 51
// cycles, and that was most of the time of a cell of thousands.  But while the
// sum stays within a binade [2^E, 2^(E+1)) its partial sums are integers P in units of
// u = 2^(E-23), and adding t = T u rounds to P + T's nearest integer, whatever P is, unless
// T is halfway: the terms round independently and the partial sums are an integer
// prefix sum.  So 128 terms are rounded at once, four per lane, and taken up to the first
// one that is large, within 2^-28 of halfway (the rounding to FP64 before shifts a sum
// by at most 2^-30 u) or brings the partial sum to the binade's ends; from there eight go
// one by one (twice as many each time that fewer than eight were taken), and on.  The sums of
// a cell of 16,276: 858,000 cycles above; the block sorter 0.24 -> 0.15 ms and the largest
// cells' 0.57 -> 0.29 ms per step of a clustered 128^3 box.  The warp sorter hides its
// chains behind one another and was slower so (85 -> 117 us).
__device__ __forceinline__ float ordered_sum(float acc, const double* x, int n) {
  const int lane = threadIdx.x & 31;
  int i = 0, single = 8;
  while (i < n) {
    const int e = (__double2hiint((double)acc) >> 20) & 0x7ff;  // E + 1023
    if (e > 900 && e < 1150) {                                  // not zero, FP32's normal range and no further
      const double scale = __hiloint2double((2069 - e) << 20, 0);  // 1 / u
      const int P0 = (int)__dmul_rn((double)acc, scale);           // exact
      int s[4], sum = 0;
      unsigned ok = 0u;
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int j = i + 4 * lane + u;
        const double T = j < n ? __dmul_rn(x[j], scale) : 1e30;
        const int r = __double2int_rn(T);
        if (fabs(T) < 4194304.0 && fabs(__dsub_rn(T, (double)r)) < 0.5 - 0x1p-28) {
          ok |= 1u << u;
          sum += r;
        }
        s[u] = sum;
      }
      int P = sum;  // at most 2^29 in all
      for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, P, o);
        if (lane >= o) P += y;
      }
      P += P0 - sum;  // the partial sum before this lane's terms
      int taken = 0;
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int a = abs(P + s[u]);
        if (taken == u && (ok >> u & 1u) && a > (1 << 23) && a < (1 << 24)) taken = u + 1;
      }
      P += taken == 0 ? 0 : taken == 1 ? s[0] : taken == 2 ? s[1] : taken == 3 ? s[2] : s[3];
      const unsigned ends = __ballot_sync(0xffffffffu, taken < 4);
      const int last = ends ? __ffs(ends) - 1 : 31;
      P = __shfl_sync(0xffffffffu, P, last);
      acc = (float)__dmul_rn((double)P, __hiloint2double((e - 23) << 20, 0));  // exact
      const int took = 4 * last + __shfl_sync(0xffffffffu, taken, last);
      i += took;
      if (!ends) continue;
      single = took < 8 ? min(2 * single, 128) : 8;
    }
    for (const int end = min(n, i + single); i < end; ++i) acc = (float)cube_dadd((double)acc, x[i]);
  }
  return acc;
}

// A tile of T keys (a power of two) in shared memory, key i at place tile_at(i): one
// place in nine stays empty, so that threads with eight neighbouring keys each meet
// different banks.
__device__ __forceinline__ int tile_at(int i) { return i + (i >> 3); }

// G successive passes of stage k of the bitonic network, strides jl 2^(G-1) .. jl, on a
// tile that starts at key `base` of the whole: a thread carries 2^G keys through them.
// Bound by the shared-memory accesses and the barriers, one of each per pass when the passes go
// one by one: a cell of 16,276 entries took 440,000 cycles to sort, three
// passes at a time in a tile that holds it 160,000 (17,473 entries, beyond the tile:
// 999,000 and 408,000); one of 4,000 in the block sorter 37,000.
template <int G>
__device__ __forceinline__ void tile_passes(unsigned long long* t, int T, int base, int jl, int k) {
  for (int p = threadIdx.x; p < (T >> G); p += blockDim.x) {
    const int i0 = ((p & ~(jl - 1)) << G) | (p & (jl - 1));
    const bool up = ((base + i0) & k) == 0;
    unsigned long long v[1 << G];
#pragma unroll
    for (int u = 0; u < (1 << G); ++u) v[u] = t[tile_at(i0 + u * jl)];
#pragma unroll
    for (int s = G - 1; s >= 0; --s)
#pragma unroll
      for (int u = 0; u < (1 << G); ++u)
        if (!((u >> s) & 1)) {
          const unsigned long long a = v[u], b = v[u | (1 << s)];
          const bool swap = (a > b) == up;
          v[u] = swap ? b : a;
          v[u | (1 << s)] = swap ? a : b;
        }
#pragma unroll
    for (int u = 0; u < (1 << G); ++u) t[tile_at(i0 + u * jl)] = v[u];
  }
  __syncthreads();
}

// the passes of stride 2^(q-1) and below of stage k, three at a time
__device__ __forceinline__ void tile_stage(unsigned long long* t, int T, int base, int q, int k) {
  for (; q >= 3; q -= 3) tile_passes<3>(t, T, base, 1 << (q - 3), k);
  if (q == 2) tile_passes<2>(t, T, base, 1, k);
  if (q == 1) tile_passes<1>(t, T, base, 1, k);
}

// ascending sort of a tile (base 0), or its stages as part of a longer one
__device__ __forceinline__ void tile_sort(unsigned long long* t, int T, int base) {
  for (int q = 1; (1 << q) <= T; ++q) tile_stage(t, T, base, q, 1 << q);
}

// The same sort for m > T keys in global memory with a shared tile of T keys
// (both powers of two): the stages up to T and, in every later stage, the passes
// of stride below T run tile by tile in shared memory; only the passes of stride
// T and above go through global memory, four compare-exchanges per thread in
// flight (their pairs are disjoint, so the loads of a batch precede its stores).
__device__ __forceinline__ void bitonic_tiled(unsigned long long* g, int m, unsigned long long* t, int T) {
  const int nthr = blockDim.x;
  for (int base = 0; base < m; base += T) {
    for (int i = threadIdx.x; i < T; i += nthr) t[tile_at(i)] = g[base + i];
    __syncthreads();
    tile_sort(t, T, base);
    for (int i = threadIdx.x; i < T; i += nthr) g[base + i] = t[tile_at(i)];
    __syncthreads();
  }
  const int npairs = m >> 1;
  for (int k = 2 * T; k <= m; k <<= 1) {
    for (int j = k >> 1; j >= T; j >>= 1) {
      for (int p0 = threadIdx.x; p0 < npairs; p0 += 4 * nthr) {
        unsigned long long a[4], bb[4];
        int ii[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int p = p0 + u * nthr;
          ii[u] = -1;
          if (p < npairs) {
            const int i = ((p & ~(j - 1)) << 1) | (p & (j - 1));  // bit j of i clear
            ii[u] = i;
            a[u] = g[i];
            bb[u] = g[i | j];
          }
        }
#pragma unroll
        for (int u = 0; u < 4; ++u)
          if (ii[u] >= 0) {
            const bool up = (ii[u] & k) == 0;
            if ((a[u] > bb[u]) == up) { g[ii[u]] = bb[u]; g[ii[u] | j] = a[u]; }
          }
      }
      __syncthreads();
    }
    for (int base = 0; base < m; base += T) {
      for (int i = threadIdx.x; i < T; i += nthr) t[tile_at(i)] = g[base + i];
      __syncthreads();
      tile_stage(t, T, base, 31 - __clz(T), k);
      for (int i = threadIdx.x; i < T; i += nthr) g[base + i] = t[tile_at(i)];
      __syncthreads();
    }
  }
}

// one crowded cell by the whole CTA: bitonic sort of (key<<32|source) (m = next power
// of two of n entries) in the shared tile of T keys, or through it in sk (global
// memory) when m > T; the sorted order back to the slots, the per-particle velocities
// into sv[d * vstride + i] (global memory) in parallel, and the FP32 sum by one warp per
// component in order, from chunks of them in the tile.
template <int ZX, int ZV>
__device__ __forceinline__ void sort_sum_cell(const RebinArgs& A, int64_t c, int n, int64_t s, unsigned long long* sk,
                                              double* sv, int vstride, unsigned long long* tile, int T) {
  int m = 1;
  while (m < n) m <<= 1;
  const bool in_tile = m <= T;
  for (int i = threadIdx.x; i < m; i += blockDim.x) {
    const unsigned long long e =
        i < n ? (((unsigned long long)A.pkey[s + i] << 32) | (uint32_t)A.perm[s + i]) : ~0ull;
    if (in_tile) tile[tile_at(i)] = e; else sk[i] = e;
  }
  __syncthreads();
  if (in_tile) tile_sort(tile, m, 0);
  else bitonic_tiled(sk, m, tile, T);
  int tt[3];
  cell_tile(A, c, tt);
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    const unsigned long long e = in_tile ? tile[tile_at(i)] : sk[i];
    const uint32_t key = (uint32_t)(e >> 32);
    const int32_t ip = (int32_t)(uint32_t)(e & 0xffffffffu);
    A.pkey[s + i] = key;  // sorted order back to the slots
    A.perm[s + i] = ip;
    const int64_t sc = src_cell(A, key, tt);
    for (int d = 0; d < 3; ++d)
      sv[(size_t)d * vstride + i] =
          cube_dadd(decode_v<ZX, ZV>(A, ip, d), (double)__ldg(&A.vfield[(size_t)d * A.ncells + sc]));
  }
  __syncthreads();
  const int d = threadIdx.x >> 5;  // a warp per component
  float acc = 0.f;
  if (d < 3) acc = (float)cube_dmul((double)A.vfield[(size_t)d * A.ncells + c], 0.1);
  double* stage = reinterpret_cast<double*>(tile);  // the keys are consumed
  const int ch = T / 3;
  for (int j0 = 0; j0 < n; j0 += ch) {
    const int len = min(ch, n - j0);
    for (int i = threadIdx.x; i < 3 * len; i += blockDim.x) {
      const int dd = i / len, k = i - dd * len;
      stage[dd * ch + k] = sv[(size_t)dd * vstride + j0 + k];
    }
    __syncthreads();
    if (d < 3) acc = ordered_sum(acc, stage + d * ch, len);
    __syncthreads();
  }
  if (d < 3 && (threadIdx.x & 31) == 0)
    A.vfield2[(size_t)d * A.ncells + c] = (float)cube_ddiv((double)acc, cube_dadd((double)n, 0.1));
  __syncthreads();
}

// the same for one cell of at most WARP_MAX entries by one warp, in the warp's
// own shared-memory segment (sk: WARP_MAX keys, sv: [3][WARP_MAX] velocities)
template <int ZX, int ZV>
__device__ __forceinline__ void sort_sum_cell_warp(const RebinArgs& A, int64_t c, int n, int64_t s, unsigned long long* sk,
                                   double* sv) {
  const int lane = threadIdx.x & 31;
  int m = 1;
  while (m < n) m <<= 1;
  for (int i = lane; i < m; i += 32)
    sk[i] = i < n ? (((unsigned long long)A.pkey[s + i] << 32) | (uint32_t)A.perm[s + i]) : ~0ull;
  __syncwarp();
  for (int k = 2; k <= m; k <<= 1)
    for (int j = k >> 1; j > 0; j >>= 1) {
      for (int i = lane; i < m; i += 32) {
        const int ixj = i ^ j;
        if (ixj > i) {
          const unsigned long long a = sk[i], bb = sk[ixj];
          const bool up = (i & k) == 0;
          if ((a > bb) == up) { sk[i] = bb; sk[ixj] = a; }
        }
      }
      __syncwarp();
    }
  int tt[3];
  cell_tile(A, c, tt);
  for (int i = lane; i < n; i += 32) {
    const uint32_t key = (uint32_t)(sk[i] >> 32);
    const int32_t ip = (int32_t)(uint32_t)(sk[i] & 0xffffffffu);
    A.pkey[s + i] = key;
    A.perm[s + i] = ip;
    const int64_t sc = src_cell(A, key, tt);
    for (int d = 0; d < 3; ++d)
      sv[d * WARP_MAX + i] = cube_dadd(decode_v<ZX, ZV>(A, ip, d), (double)__ldg(&A.vfield[(size_t)d * A.ncells + sc]));
  }
  __syncwarp();
  if (lane < 3) {
    const int d = lane;
    const float acc = ordered_sum_lane((float)cube_dmul((double)A.vfield[(size_t)d * A.ncells + c], 0.1),
                                       sv + d * WARP_MAX, n);
    A.vfield2[(size_t)d * A.ncells + c] = (float)cube_ddiv((double)acc, cube_dadd((double)n, 0.1));
  }
  __syncwarp();
}

// F1 for cells of SMALL+1..WARP_MAX entries: one warp per cell
template <int ZX, int ZV>
__global__ void __launch_bounds__(32 * WARP_WARPS) k_rebin_warp(RebinArgs A) {
  extern __shared__ unsigned long long wsm[];
  const int w = threadIdx.x >> 5;
  unsigned long long* sk = wsm + (size_t)w * 4 * WARP_MAX;
  double* sv = reinterpret_cast<double*>(sk + WARP_MAX);
  const unsigned long long nw = A.dscal->n_big;
  const unsigned long long stride = (unsigned long long)gridDim.x * WARP_WARPS;
  for (unsigned long long b = (unsigned long long)blockIdx.x * WARP_WARPS + w; b < nw; b += stride) {
    const int64_t c = A.big_list[b];
    sort_sum_cell_warp<ZX, ZV>(A, c, A.cnt2[c], A.start2[c], sk, sv);
  }
}

// F1 for cells of WARP_MAX+1..BIG_MAX entries: one CTA per cell, keys sorted in
// shared memory (36 KB, so that several CTAs share an SM and their barriers overlap),
// the velocity columns in the CTA's global slot of 3 BIG_MAX doubles; cells are
// taken as CTAs become free
template <int ZX, int ZV>
__global__ void __launch_bounds__(512) k_rebin_big(RebinArgs A, double* __restrict__ scratch) {
  extern __shared__ unsigned long long tile[];
  __shared__ unsigned long long qs;
  double* sv = scratch + (size_t)blockIdx.x * 3 * BIG_MAX;
  const unsigned long long nmid = A.dscal->n_mid;
  while (true) {
    if (threadIdx.x == 0) qs = atomicAdd(&A.dscal->mid_next, 1ull);
    __syncthreads();
    const unsigned long long b = qs;
    __syncthreads();
    if (b >= nmid) break;
    const int64_t c = A.big_list[A.ncells - 1 - (int64_t)b];
    sort_sum_cell<ZX, ZV>(A, c, A.cnt2[c], A.start2[c], nullptr, sv, BIG_MAX, tile, BIG_MAX);
  }
}

// F1 for cells beyond BIG_MAX: the same in a global scratch slot per CTA
// (slot_u64 = keys for the largest cell padded to a power of two, then its
// velocities)
constexpr int HUGE_TILE = 16384;  // keys per shared tile of the huge-cell sort (144 KB)
template <int ZX, int ZV>
__global__ void __launch_bounds__(1024) k_rebin_huge(RebinArgs A, unsigned long long* __restrict__ scratch,
                                                     size_t slot_u64, int mmax) {
  extern __shared__ unsigned long long tile[];
  __shared__ unsigned long long qs;
  unsigned long long* sk = scratch + (size_t)blockIdx.x * slot_u64;
  double* sv = reinterpret_cast<double*>(sk + mmax);
  const unsigned long long nh = A.dscal->n_huge;
  const int vstride = (int)((slot_u64 - mmax) / 3);
  while (true) {  // cells taken in list order (largest first) as blocks become free
    if (threadIdx.x == 0) qs = atomicAdd(&A.dscal->huge_next, 1ull);
    __syncthreads();
    const unsigned long long q = qs;
    __syncthreads();
    if (q >= nh) break;
    const int64_t c = A.cursor[q];
    sort_sum_cell<ZX, ZV>(A, c, A.cnt2[c], A.start2[c], sk, sv, vstride, tile, HUGE_TILE);
  }
}

// the huge-cell list in decreasing particle count (bitonic sort of (~n, cell) in
// shared memory), so that the largest cells start first; lists longer than
// HUGE_ORDER stay in arrival order
constexpr int HUGE_ORDER = 4096;
__global__ void __launch_bounds__(1024) k_rebin_huge_order(RebinArgs A) {
  __shared__ unsigned long long h[HUGE_ORDER];
  const int nh = (int)A.dscal->n_huge;
  if (nh < 2 || nh > HUGE_ORDER) return;
  int m = 1;
  while (m < nh) m <<= 1;
  for (int i = threadIdx.x; i < m; i += blockDim.x) {
    if (i < nh) {
      const int32_t c = A.cursor[i];
      h[i] = ((unsigned long long)(~(uint32_t)A.cnt2[c]) << 32) | (uint32_t)c;
    } else {
      h[i] = ~0ull;
    }
  }
  __syncthreads();
  for (int k = 2; k <= m; k <<= 1)
    for (int j = k >> 1; j > 0; j >>= 1) {
      for (int i = threadIdx.x; i < m; i += blockDim.x) {
        const int ixj = i ^ j;
        if (ixj > i) {
          const unsigned long long a = h[i], bb = h[ixj];
          const bool up = (i & k) == 0;
          if ((a > bb) == up) { h[i] = bb; h[ixj] = a; }
        }
      }
      __syncthreads();
    }
  for (int i = threadIdx.x; i < nh; i += blockDim.x) A.cursor[i] = (int32_t)(uint32_t)(h[i] & 0xffffffffu);
}

// F2: the entries of the crowded cells, sorted in their slots by the sorters, one
// thread per entry over work items of the new layout (so that a cell of many thousand
// entries is shared by several CTAs)
template <int ZX, int ZV>
__global__ void __launch_bounds__(256) k_rebin_emit(RebinArgs A) {
  __shared__ int64_t cs[RCELLS];
  __shared__ uint8_t big[RCELLS];
  int64_t c0, p0, p1;
  int ncl;
  if (!get_item(A, c0, ncl, p0, p1)) return;
  int crowded = 0;
  for (int i = threadIdx.x; i < ncl; i += blockDim.x) {
    const int n = A.cnt2[c0 + i];
    cs[i] = A.start2[c0 + i];
    big[i] = n > SMALL;
    crowded |= n > SMALL;
  }
  if (!__syncthreads_or(crowded)) return;
  for (int64_t s = p0 + threadIdx.x; s < p1; s += blockDim.x) {
    int lo = 0, hi = ncl - 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (cs[mid] <= s) lo = mid; else hi = mid - 1;
    }
    if (!big[lo]) continue;
    const int64_t c = c0 + lo;
    int tt[3];
    cell_tile(A, c, tt);
    const int32_t ip = A.perm[s];
    double v[3];
    entry_velocity<ZV>(A, A.pkey[s], ip, tt, v);
    const float m[3] = {A.vfield2[c], A.vfield2[A.ncells + c], A.vfield2[2 * A.ncells + c]};
    emit_one<ZX, ZV>(A, c, s, ip, v, m);
  }
}

template <int ZX, int ZV>
int run_rebin(cube_ctx* ctx, RebinArgs& A) {
  CUBE_CUDA_TRY(ctx, cudaMemsetAsync(ctx->rhoc2, 0, sizeof(int32_t) * ctx->ncells, ctx->stream));
  int64_t ni = 0;  // one block per item (blocks past the last item return at once)
  int rc = cube_cell_items(ctx, ctx->cell_start, ctx->cells_le32, &A.items, &ni);
  if (rc) return rc;
  k_rebin_count<ZX, ZV><<<(unsigned)ni, 256, 0, ctx->stream>>>(A);
  CUBE_LAUNCH_CHECK(ctx);
  rc = cube_exclusive_scan(ctx, A.cnt2, ctx->ncells, A.start2, &ctx->dscal->np_new, A.cursor);  // and the cursors zero
  if (rc) return rc;
  k_rebin_place<<<1184, 256, 0, ctx->stream>>>(A, ctx->np);
  CUBE_LAUNCH_CHECK(ctx);
  k_rebin_cells<ZX, ZV><<<(unsigned)((ctx->ncells + GCELLS - 1) / GCELLS), GTHREADS, 0, ctx->stream>>>(A);
  CUBE_LAUNCH_CHECK(ctx);
  return CUBE_OK;
}

// the crowded cells, from the lists' sizes in hscal
template <int ZX, int ZV>
int run_rebin_crowded(cube_ctx* ctx, RebinArgs& A) {
  // n_huge, max_huge, n_mid, n_big
  const unsigned long long hv[4] = {ctx->hscal->n_huge, ctx->hscal->max_huge, ctx->hscal->n_mid, ctx->hscal->n_big};
  // Cells beyond the block sorter first, on a stream beside the context's: few CTAs whose
  // time is the largest cell's, while the other sorters fill the GPU (four steps of a
  // clustered 128^3 box: 10.7 ms one after the other, 9.3 ms so).
  int rc = CUBE_OK;
  if (hv[0]) {
    // one slot per SM of keys (mmax, a power of two) and three velocity columns
    // of mmax: the scratch is reallocated only when mmax doubles
    int mmax = 1;
    while ((unsigned long long)mmax < hv[1]) mmax <<= 1;
    const size_t slot = 4 * (size_t)mmax;
    const int grid = (int)std::min<unsigned long long>(hv[0], (unsigned long long)ctx->num_sms);
    const size_t need = sizeof(unsigned long long) * slot * ctx->num_sms;
    if (need > ctx->rebin_scratch_bytes) {
      if (ctx->rebin_scratch) cudaFree(ctx->rebin_scratch);
      ctx->rebin_scratch = nullptr;
      ctx->rebin_scratch_bytes = 0;
      CUBE_CUDA_TRY(ctx, cudaMalloc(&ctx->rebin_scratch, need));
      ctx->rebin_scratch_bytes = need;
    }
    const size_t tsmem = sizeof(unsigned long long) * (HUGE_TILE + HUGE_TILE / 8);
    CUBE_CUDA_TRY(ctx, cube_smem_limit(ctx, k_rebin_huge<ZX, ZV>, tsmem));
    if (!ctx->side) {
      CUBE_CUDA_TRY(ctx, cudaStreamCreateWithFlags(&ctx->side, cudaStreamNonBlocking));
      for (cudaEvent_t& e : ctx->side_ev) CUBE_CUDA_TRY(ctx, cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
    }
    CUBE_CUDA_TRY(ctx, cudaEventRecord(ctx->side_ev[0], ctx->stream));
    CUBE_CUDA_TRY(ctx, cudaStreamWaitEvent(ctx->side, ctx->side_ev[0], 0));
    // (an error from here on still waits for the side stream)
    rc = [&]() -> int {
      k_rebin_huge_order<<<1, 1024, 0, ctx->side>>>(A);
      CUBE_LAUNCH_CHECK(ctx);
      k_rebin_huge<ZX, ZV><<<grid, 1024, tsmem, ctx->side>>>(
          A, reinterpret_cast<unsigned long long*>(ctx->rebin_scratch), slot, mmax);
      CUBE_LAUNCH_CHECK(ctx);
      return CUBE_OK;
    }();
  }
  if (!rc) rc = [&]() -> int {
    if (hv[3]) {
      const size_t wsmem = sizeof(unsigned long long) * 4 * WARP_MAX * WARP_WARPS;
      CUBE_CUDA_TRY(ctx, cube_smem_limit(ctx, k_rebin_warp<ZX, ZV>, wsmem));
      k_rebin_warp<ZX, ZV><<<3 * ctx->num_sms, 32 * WARP_WARPS, wsmem, ctx->stream>>>(A);
      CUBE_LAUNCH_CHECK(ctx);
    }
    if (hv[2]) {
      const int nblk = 4 * ctx->num_sms;
      if (!ctx->rebin_mid_scratch)
        CUBE_CUDA_TRY(ctx, cudaMalloc(&ctx->rebin_mid_scratch, sizeof(double) * 3 * BIG_MAX * (size_t)nblk));
      const size_t smem = sizeof(unsigned long long) * (BIG_MAX + BIG_MAX / 8);
      CUBE_CUDA_TRY(ctx, cube_smem_limit(ctx, k_rebin_big<ZX, ZV>, smem));
      const int grid = (int)std::min<unsigned long long>(hv[2], (unsigned long long)nblk);
      k_rebin_big<ZX, ZV><<<grid, 512, smem, ctx->stream>>>(A, reinterpret_cast<double*>(ctx->rebin_mid_scratch));
      CUBE_LAUNCH_CHECK(ctx);
    }
    return CUBE_OK;
  }();
  if (hv[0]) {
    cudaError_t e = cudaEventRecord(ctx->side_ev[1], ctx->side);
    if (e == cudaSuccess) e = cudaStreamWaitEvent(ctx->stream, ctx->side_ev[1], 0);
    if (e != cudaSuccess) cudaStreamSynchronize(ctx->side);
    CUBE_CUDA_TRY(ctx, e);
  }
  if (rc) return rc;
  // their entries, over work items of the new layout
  int64_t ni = 0;
  rc = cube_cell_items(ctx, A.start2, false, &A.items, &ni);
  if (rc) return rc;
  k_rebin_emit<ZX, ZV><<<(unsigned)ni, 256, 0, ctx->stream>>>(A);
  CUBE_LAUNCH_CHECK(ctx);
  return CUBE_OK;
}

}  // namespace

int64_t cube_rebin_items_max(int64_t ncells, int64_t cap) {
  return (ncells + RCELLS - 1) / RCELLS + 4 * (cap / PMAX + 1) + 64;
}

int cube_cell_items(cube_ctx* ctx, const int64_t* cell_start, bool le32, const int64_t** items, int64_t* blocks) {
  const int64_t ngroups = (ctx->ncells + RCELLS - 1) / RCELLS;
  *items = nullptr;
  *blocks = ngroups;
  if (le32) return CUBE_OK;  // at most 32 RCELLS <= PMAX particles in a group
  const int64_t items_max = cube_rebin_items_max(ctx->ncells, ctx->cap);
  CUBE_CUDA_TRY(ctx, cudaMemsetAsync(&ctx->dscal->n_items, 0, sizeof(unsigned long long), ctx->stream));
  k_cell_items<<<(unsigned)((ngroups + 255) / 256), 256, 0, ctx->stream>>>(cell_start, ctx->ncells, ctx->rebin_items,
                                                                         items_max, ctx->dscal);
  CUBE_LAUNCH_CHECK(ctx);
  *items = ctx->rebin_items;
  *blocks = std::min<int64_t>(items_max, ngroups + 4 * (ctx->np / PMAX + 1));
  return CUBE_OK;
}

int cube_rebin(cube_ctx* ctx, cube_scalars* io, bool crowded) {
  io->dt_mid = (io->dt_old + io->dt) / 2;
  const float q = cube_fdiv(cube_fmul(io->dt_mid, io->vz_max), (float)ctx->ncell);
  const int nlayer = 2 * (int)ceilf(q) + 1;
  io->nlayer = nlayer;
  RebinArgs A;
  A.xp = ctx->xp; A.vp = ctx->vp; A.pid = ctx->pid;
  A.cell_start = ctx->cell_start; A.vfield = ctx->vfield;
  A.xp2 = ctx->xp2; A.vp2 = ctx->vp2; A.pid2 = ctx->pid2;
  A.cnt2 = ctx->rhoc2; A.start2 = ctx->cell_start2; A.vfield2 = ctx->vfield2;
  A.tcell = ctx->tcell; A.tkey = ctx->tkey; A.perm = ctx->perm; A.pkey = ctx->pkey; A.cursor = ctx->cursor;
  A.big_list = ctx->big_list;
  A.items = nullptr; A.items_max = cube_rebin_items_max(ctx->ncells, ctx->cap);
  A.slot_cell = reinterpret_cast<int32_t*>(ctx->slot_r2);
  A.half_nvbin = ctx->nvbin / 2;
  A.codec = ctx->codec; A.coef = cube_vcoef(&ctx->codec, io->sigma_vi);
  A.tab = cube_venc_tab(ctx);
  {
    int trc;
    A.dec = cube_vdec_table(ctx, A.coef, &trc);
    if (trc) return trc;
  }
  A.cap = ctx->cap; A.ncells = ctx->ncells;
  A.nc = ctx->nc; A.nt = ctx->nt; A.nnt = ctx->nnt; A.ncb = ctx->ncb; A.nte = ctx->nte; A.ncell = ctx->ncell;
  A.nlayer = nlayer; A.use_pid = ctx->P.use_pid; A.dt_mid = io->dt_mid; A.dscal = ctx->dscal;
  A.dnt = cube_fastdiv(ctx->nt);
  A.dnt3 = cube_fastdiv((uint32_t)ctx->nt * ctx->nt * ctx->nt);
  A.dnnt = cube_fastdiv(ctx->nnt);
  A.dnlayer = cube_fastdiv(nlayer);
  A.dnte = cube_fastdiv(ctx->nte, (uint64_t)nlayer * ctx->nte * ctx->nte * ctx->nte >= (uint64_t)1 << 31);
  A.inv_ncell = 1.0 / (double)ctx->ncell;
  A.inv_xstep = 1.0 / (ctx->codec.x_resolution * (double)ctx->ncell);
  {
    int e1, e2;  // both divisors must be powers of two for the products to equal the quotients
    if (std::frexp((double)ctx->ncell, &e1) != 0.5 || std::frexp(ctx->codec.x_resolution * ctx->ncell, &e2) != 0.5) {
      ctx->err = "re-bin: ncell and x_resolution*ncell must be powers of two";
      return CUBE_ERR_PARAM;
    }
  }
  const int zx = ctx->izipx, zv = ctx->izipv;
  if (crowded) {
    if (zx == 1) return zv == 1 ? run_rebin_crowded<1, 1>(ctx, A) : run_rebin_crowded<1, 2>(ctx, A);
    return zv == 1 ? run_rebin_crowded<2, 1>(ctx, A) : run_rebin_crowded<2, 2>(ctx, A);
  }
  if (zx == 1) return zv == 1 ? run_rebin<1, 1>(ctx, A) : run_rebin<1, 2>(ctx, A);
  return zv == 1 ? run_rebin<2, 1>(ctx, A) : run_rebin<2, 2>(ctx, A);
}
