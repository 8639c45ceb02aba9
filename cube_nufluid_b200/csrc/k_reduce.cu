/*
 * k_reduce.cu -- deterministic reductions and the cell-count prefix scan.
 *
 * cube_tree_sum_dev: the sum of n doubles as a fixed pairwise tree over
 * blocks of 1024 (pad with zeros; loc[i] += loc[i+s] for s = 512..1), then
 * the same tree over the block sums, until one value is left.  The CPU
 * oracle uses the identical tree, so sums such as the velocity statistics of
 * update_x (update_particle.f90:174-226) agree to the last bit.
 *
 * cube_exclusive_scan: int32 cell counts -> int64 cell starts (n+1 entries),
 * the role of spine_tile / spine_image (variables.f90:103-218).
 */
#include "cube_internal.cuh"

namespace {

// one level of the tree; blockIdx.y: which of several arrays
__global__ void k_tree_block(const double* __restrict__ in, int64_t n, int64_t in_stride, double* __restrict__ out,
                             int64_t out_stride) {
  __shared__ double loc[512];
  in += blockIdx.y * in_stride;
  out += blockIdx.y * out_stride;
  const int i = threadIdx.x;  // 512 threads
  const int64_t b = blockIdx.x;
  const int64_t q0 = b * 1024 + i, q1 = q0 + 512;
  const double a0 = q0 < n ? in[q0] : 0.0;
  const double a1 = q1 < n ? in[q1] : 0.0;
  loc[i] = __dadd_rn(a0, a1);  // s = 512
  __syncthreads();
  for (int s = 256; s >= 32; s >>= 1) {
    if (i < s) loc[i] = __dadd_rn(loc[i], loc[i + s]);
    __syncthreads();
  }
  if (i < 32) {
    double v = loc[i];
    for (int s = 16; s >= 1; s >>= 1) {
      const double o = __shfl_down_sync(0xffffffffu, v, s);
      if (i < s) v = __dadd_rn(v, o);
    }
    if (i == 0) out[b] = v;
  }
}

// The first level of the tree over the per-particle velocity statistics of update_x
// (update_particle.f90:174-226) with the terms formed here: for slot q of the new
// storage order, vr = tan(code)/coef of its new residual code and vs = vr + vfield of
// its new cell, r2 = (vr_x^2 + vr_y^2) + vr_z^2 and s2 likewise from vs; the two
// block sums follow the tree of k_tree_block exactly, so the totals are the ones a
// stored list of terms would give (0 past the end).
// One CTA of 256 threads per 1024-block of the tree, the same additions in the same
// order as k_tree_block: thread i forms elements i, i+256, i+512, i+768 (all their reads
// in flight together), the stages of stride 512 and 256 are its own, and one warp per
// quantity does the rest: lane l holds 32w + l, w = 0..7 (strides 128, 64, 32 in
// registers), then the same shuffles.  Bound by the latency of the dependent reads
// (codes and cell, then decode table and cell mean): a warp per block with 32
// elements per lane in turn took 24 us for the 32 blocks of 32^3 particles,
// this 4.7 us.
// one block b by the 256 threads i, with dec(code) the decode; sync() joins the threads
template <int ZV, typename Dec, typename Sync>
__device__ __forceinline__ void stats_block(const void* __restrict__ vp_, int64_t cap,
                                            const int32_t* __restrict__ slot_cell, const float* __restrict__ vfield,
                                            int64_t ncells, int64_t n, double* __restrict__ out_r,
                                            double* __restrict__ out_s, int64_t b, int i, double loc[2][256],
                                            const Dec& dec, const Sync& sync) {
  typedef typename CodeT<ZV>::T TV;
  const TV* vp = reinterpret_cast<const TV*>(vp_);
  const int64_t base = b * 1024 + i;
  int64_t c[4];
  int code[4][3];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int64_t q = min(base + 256 * k, n - 1);
    c[k] = slot_cell[q];
    // a crowded cell's slot is written after the others' (never read as a result before)
    if ((uint64_t)c[k] >= (uint64_t)ncells) c[k] = 0;
#pragma unroll
    for (int d = 0; d < 3; ++d) code[k][d] = (int)vp[(size_t)d * cap + q];
  }
  double r[4], s[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    r[k] = 0.0;
    s[k] = 0.0;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      const double vr = dec(code[k][d]);
      const double vs = __dadd_rn(vr, (double)__ldg(&vfield[(size_t)d * ncells + c[k]]));
      r[k] = __dadd_rn(r[k], __dmul_rn(vr, vr));
      s[k] = __dadd_rn(s[k], __dmul_rn(vs, vs));
    }
    if (base + 256 * k >= n) r[k] = s[k] = 0.0;
  }
  loc[0][i] = __dadd_rn(__dadd_rn(r[0], r[2]), __dadd_rn(r[1], r[3]));
  loc[1][i] = __dadd_rn(__dadd_rn(s[0], s[2]), __dadd_rn(s[1], s[3]));
  sync();
  const int w = i >> 5, lane = i & 31;
  if (w >= 2) return;
  double v[8];
#pragma unroll
  for (int k = 0; k < 8; ++k) v[k] = loc[w][32 * k + lane];
#pragma unroll
  for (int h = 4; h >= 1; h >>= 1)  // strides 128, 64, 32
#pragma unroll
    for (int k = 0; k < h; ++k) v[k] = __dadd_rn(v[k], v[k + h]);
  for (int o = 16; o >= 1; o >>= 1) {
    const double x = __shfl_down_sync(0xffffffffu, v[0], o);
    if (lane < o) v[0] = __dadd_rn(v[0], x);
  }
  if (lane == 0) (w ? out_s : out_r)[b] = v[0];
}

template <int ZV>
__global__ void __launch_bounds__(256) k_stats_first(const void* __restrict__ vp, int64_t cap,
                                                     const int32_t* __restrict__ slot_cell,
                                                     const float* __restrict__ vfield, int64_t ncells,
                                                     const double* __restrict__ dec, int half_nvbin, int64_t n,
                                                     double* __restrict__ out_r, double* __restrict__ out_s) {
  __shared__ double loc[2][256];
  stats_block<ZV>(vp, cap, slot_cell, vfield, ncells, n, out_r, out_s, blockIdx.x, threadIdx.x, loc,
                  [&](int code) { return __ldg(&dec[code + half_nvbin]); }, []() { __syncthreads(); });
}

constexpr int64_t STATS_P_MIN = 1 << 23;  // particles from which k_stats_p is taken
// The same with one CTA of 1024 threads per SM, each 256 of them taking every
// 4 gridDim-th block: the decodes, 96 of the 110 or so L1 lines that a warp reads,
// come from the tangents in shared memory.  loc is used in turn, so that the six warps
// without a part in the tail go on to the next block (who writes a buffer again has
// passed the barrier that the tail's warps reach after they read it).  512^3 particles:
// 1.29 ms with the tables, 0.60 so; 256^3: 166 and 95 us; 160^3, where the tangents' load is
// still felt: 34.0 and 36.2 us, and so the rule.
template <int ZV>
__global__ void __launch_bounds__(1024, 1) k_stats_p(const void* __restrict__ vp, int64_t cap,
                                                     const int32_t* __restrict__ slot_cell,
                                                     const float* __restrict__ vfield, int64_t ncells,
                                                     const float* __restrict__ tan_table, int half, double coef,
                                                     double rcp, int64_t n, int64_t nb, double* __restrict__ out_r,
                                                     double* __restrict__ out_s) {
  extern __shared__ float tan_s[];  // [half + 1]
  __shared__ double loc[4][2][2][256];
  cube_tan_load(tan_s, tan_table, half);
  __syncthreads();
  const int g = threadIdx.x >> 8;
  int turn = 0;
  for (int64_t b = 4 * (int64_t)blockIdx.x + g; b < nb; b += 4 * (int64_t)gridDim.x, turn ^= 1)
    stats_block<ZV>(vp, cap, slot_cell, vfield, ncells, n, out_r, out_s, b, threadIdx.x & 255, loc[g][turn],
                    [&](int code) { return cube_div_rcp(cube_tan_of(tan_s, code), coef, rcp); },
                    [&]() { asm volatile("bar.sync %0, 256;" ::"r"(1 + g) : "memory"); });
}

// the first level over the cells' |vfield|^2 (FP32 terms, update_particle.f90:183)
__device__ __forceinline__ double vf2(const float* __restrict__ vfield, int64_t ncells, int64_t c) {
  if (c >= ncells) return 0.0;
  const float x = vfield[c], y = vfield[ncells + c], z = vfield[2 * ncells + c];
  return (double)cube_fadd(cube_fadd(cube_fmul(x, x), cube_fmul(y, y)), cube_fmul(z, z));
}
__global__ void __launch_bounds__(512) k_vfield_first(const float* __restrict__ vfield, int64_t ncells,
                                                      double* __restrict__ out) {
  __shared__ double loc[512];
  const int i = threadIdx.x;
  const int64_t q = (int64_t)blockIdx.x * 1024 + i;
  loc[i] = __dadd_rn(vf2(vfield, ncells, q), vf2(vfield, ncells, q + 512));
  __syncthreads();
  for (int s = 256; s >= 32; s >>= 1) {
    if (i < s) loc[i] = __dadd_rn(loc[i], loc[i + s]);
    __syncthreads();
  }
  if (i < 32) {
    double v = loc[i];
    for (int s = 16; s >= 1; s >>= 1) {
      const double o = __shfl_down_sync(0xffffffffu, v, s);
      if (i < s) v = __dadd_rn(v, o);
    }
    if (i == 0) out[blockIdx.x] = v;
  }
}

constexpr int SCAN_PER_THREAD = 8;
constexpr int SCAN_THREADS = 256;
constexpr int SCAN_BLOCK = SCAN_PER_THREAD * SCAN_THREADS;

__global__ void k_scan_sums(const int32_t* __restrict__ in, int64_t n, int64_t* __restrict__ bsum) {
  __shared__ int64_t ws[32];
  const int64_t base = (int64_t)blockIdx.x * SCAN_BLOCK + threadIdx.x * SCAN_PER_THREAD;
  int64_t s = 0;
  for (int k = 0; k < SCAN_PER_THREAD; ++k)
    if (base + k < n) s += in[base + k];
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    int64_t t = 0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += ws[w];
    bsum[blockIdx.x] = t;
  }
}

// exclusive scan of nb values in place by one block
__global__ void k_scan_top(int64_t* __restrict__ v, int64_t nb) {
  __shared__ int64_t carry;
  __shared__ int64_t ws[32];
  if (threadIdx.x == 0) carry = 0;
  __syncthreads();
  for (int64_t base = 0; base < nb; base += blockDim.x) {
    const int64_t q = base + threadIdx.x;
    const int64_t x = q < nb ? v[q] : 0;
    int64_t inc = x;
    for (int o = 1; o < 32; o <<= 1) {
      const int64_t y = __shfl_up_sync(0xffffffffu, inc, o);
      if ((threadIdx.x & 31) >= o) inc += y;
    }
    if ((threadIdx.x & 31) == 31) ws[threadIdx.x >> 5] = inc;
    __syncthreads();
    if (threadIdx.x < 32) {
      const int nw = blockDim.x >> 5;
      int64_t w = threadIdx.x < nw ? ws[threadIdx.x] : 0;
      for (int o = 1; o < 32; o <<= 1) {
        const int64_t y = __shfl_up_sync(0xffffffffu, w, o);
        if ((int)threadIdx.x >= o) w += y;
      }
      ws[threadIdx.x] = w;  // inclusive warp totals
    }
    __syncthreads();
    const int wi = threadIdx.x >> 5;
    const int64_t before = (wi ? ws[wi - 1] : 0) + carry;
    if (q < nb) v[q] = before + inc - x;
    __syncthreads();
    if (threadIdx.x == blockDim.x - 1) carry = before + inc;
    __syncthreads();
  }
}

__global__ void k_scan_apply(const int32_t* __restrict__ in, int64_t n, const int64_t* __restrict__ boff,
                             int64_t* __restrict__ out, long long* __restrict__ total, int32_t* __restrict__ zero) {
  __shared__ int64_t ws[32];
  const int64_t base = (int64_t)blockIdx.x * SCAN_BLOCK + threadIdx.x * SCAN_PER_THREAD;
  int64_t vals[SCAN_PER_THREAD];
  int64_t s = 0;
  for (int k = 0; k < SCAN_PER_THREAD; ++k) {
    vals[k] = (base + k < n) ? in[base + k] : 0;
    s += vals[k];
  }
  int64_t inc = s;
  for (int o = 1; o < 32; o <<= 1) {
    const int64_t y = __shfl_up_sync(0xffffffffu, inc, o);
    if ((threadIdx.x & 31) >= o) inc += y;
  }
  if ((threadIdx.x & 31) == 31) ws[threadIdx.x >> 5] = inc;
  __syncthreads();
  if (threadIdx.x < 32) {
    const int nw = blockDim.x >> 5;
    int64_t w = threadIdx.x < nw ? ws[threadIdx.x] : 0;
    for (int o = 1; o < 32; o <<= 1) {
      const int64_t y = __shfl_up_sync(0xffffffffu, w, o);
      if ((int)threadIdx.x >= o) w += y;
    }
    ws[threadIdx.x] = w;
  }
  __syncthreads();
  const int wi = threadIdx.x >> 5;
  int64_t run = boff[blockIdx.x] + (wi ? ws[wi - 1] : 0) + inc - s;
  for (int k = 0; k < SCAN_PER_THREAD; ++k) {
    if (base + k < n) {
      out[base + k] = run;
      if (zero) zero[base + k] = 0;
    }
    run += vals[k];
  }
  if (blockIdx.x == gridDim.x - 1 && threadIdx.x == blockDim.x - 1) {
    out[n] = boff[blockIdx.x] + ws[(blockDim.x >> 5) - 1];
    if (total) *total = out[n];
  }
}

// the whole scan of at most SCAN_ONE counts in one block, up to 8 neighbouring counts per
// thread, read together.  A small box's scan is three launches otherwise, and their
// gaps most of it; beyond 8 counts per thread the block's own time is what counts.
constexpr int64_t SCAN_ONE = 8192;
__global__ void __launch_bounds__(1024) k_scan_one(const int32_t* __restrict__ in, int n, int64_t* __restrict__ out,
                                                   long long* __restrict__ total, int32_t* __restrict__ zero) {
  __shared__ int64_t ws[32];
  const int per = (n + 1023) / 1024, b = (int)threadIdx.x * per;
  int v[SCAN_ONE / 1024];
  int64_t s = 0;
#pragma unroll
  for (int k = 0; k < SCAN_ONE / 1024; ++k) v[k] = k < per && b + k < n ? in[b + k] : 0;
#pragma unroll
  for (int k = 0; k < SCAN_ONE / 1024; ++k) s += v[k];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  int64_t inc = s;
  for (int o = 1; o < 32; o <<= 1) {
    const int64_t y = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += y;
  }
  if (lane == 31) ws[w] = inc;
  __syncthreads();
  if (w == 0) {
    int64_t t = ws[lane];
    for (int o = 1; o < 32; o <<= 1) {
      const int64_t y = __shfl_up_sync(0xffffffffu, t, o);
      if (lane >= o) t += y;
    }
    ws[lane] = t;
  }
  __syncthreads();
  int64_t run = (w ? ws[w - 1] : 0) + inc - s;
#pragma unroll
  for (int k = 0; k < SCAN_ONE / 1024; ++k) {
    if (k < per && b + k < n) {
      out[b + k] = run;
      if (zero) zero[b + k] = 0;
    }
    run += v[k];
  }
  if (threadIdx.x == 1023) {
    out[n] = ws[31];
    if (total) *total = ws[31];
  }
}

}  // namespace

int cube_stats_sums(cube_ctx* ctx, const int32_t* slot_cell, const double* dec, double coef) {
  const int64_t n = ctx->np;
  double* out = ctx->dscal->sums;
  // block sums in the per-slot array, free after the re-bin, and of the cells in theirs
  const int64_t nbc = (ctx->ncells + 1023) / 1024;
  k_vfield_first<<<(unsigned)nbc, 512, 0, ctx->stream>>>(ctx->vfield2, ctx->ncells, ctx->cell_stats);
  CUBE_LAUNCH_CHECK(ctx);
  int rc = cube_tree_sums_async(ctx, ctx->cell_stats, nbc, 0, 1, out);
  if (rc || n == 0) return rc;  // DevScal is zero at the start of the call
  const int64_t nb = (n + 1023) / 1024;
  double* br = ctx->slot_s2;
  if (cube_use_tan(ctx, coef) && n >= STATS_P_MIN) {
    const int half = ctx->nvbin / 2;
    const size_t smem = sizeof(float) * ((size_t)half + 1);
    auto k = ctx->izipv == 1 ? k_stats_p<1> : k_stats_p<2>;
    CUBE_CUDA_TRY(ctx, cube_smem_limit(ctx, k, smem));
    k<<<ctx->num_sms, 1024, smem, ctx->stream>>>(ctx->vp2, ctx->cap, slot_cell, ctx->vfield2, ctx->ncells,
                                                 ctx->tan_table, half, coef, 1.0 / coef, n, nb, br, br + nb);
  } else {
    auto k = ctx->izipv == 1 ? k_stats_first<1> : k_stats_first<2>;
    k<<<(unsigned)nb, 256, 0, ctx->stream>>>(ctx->vp2, ctx->cap, slot_cell, ctx->vfield2, ctx->ncells, dec,
                                             ctx->nvbin / 2, n, br, br + nb);
  }
  CUBE_LAUNCH_CHECK(ctx);
  return cube_tree_sums_async(ctx, br, nb, nb, 2, out + 1);
}

int cube_tree_sums_async(cube_ctx* ctx, const double* in, int64_t n, int64_t stride, int count, double* out_dev) {
  double* bufs[2];
  const int64_t half = (n + 1023) / 1024;
  bufs[0] = ctx->red_tmp;
  bufs[1] = ctx->red_tmp + count * half;
  const double* src = in;
  int64_t m = n, st = stride;
  for (int flip = 0;; flip ^= 1) {
    const int64_t nb = (m + 1023) / 1024;
    double* dst = nb == 1 ? out_dev : bufs[flip];
    k_tree_block<<<dim3((unsigned)nb, count), 512, 0, ctx->stream>>>(src, m, st, dst, nb);
    CUBE_LAUNCH_CHECK(ctx);
    if (nb == 1) return CUBE_OK;
    src = dst;
    m = st = nb;
  }
}

int cube_tree_sum_dev(cube_ctx* ctx, const double* in, int64_t n, double* out_host) {
  if (n == 0) { *out_host = 0.0; return CUBE_OK; }
  double* out = ctx->red_tmp + (n + 1023) / 1024 * 2;  // past the levels' buffers
  const int rc = cube_tree_sums_async(ctx, in, n, 0, 1, out);
  if (rc) return rc;
  CUBE_CUDA_TRY(ctx, cudaMemcpyAsync(out_host, out, sizeof(double), cudaMemcpyDeviceToHost, ctx->stream));
  CUBE_CUDA_TRY(ctx, cudaStreamSynchronize(ctx->stream));
  return CUBE_OK;
}

int cube_exclusive_scan(cube_ctx* ctx, const int32_t* in, int64_t n, int64_t* out, long long* total, int32_t* zero) {
  if (n <= SCAN_ONE) {
    k_scan_one<<<1, 1024, 0, ctx->stream>>>(in, (int)n, out, total, zero);
    CUBE_LAUNCH_CHECK(ctx);
    return CUBE_OK;
  }
  const int64_t nb = (n + SCAN_BLOCK - 1) / SCAN_BLOCK;
  int64_t* bs = ctx->scan_tmp;
  k_scan_sums<<<(unsigned)nb, SCAN_THREADS, 0, ctx->stream>>>(in, n, bs);
  CUBE_LAUNCH_CHECK(ctx);
  k_scan_top<<<1, 1024, 0, ctx->stream>>>(bs, nb);
  CUBE_LAUNCH_CHECK(ctx);
  k_scan_apply<<<(unsigned)nb, SCAN_THREADS, 0, ctx->stream>>>(in, n, bs, out, total, zero);
  CUBE_LAUNCH_CHECK(ctx);
  return CUBE_OK;
}

namespace {
// decode of every code, one bit per code: the step's encode returns the code itself for
// its decoded velocity, and per block (one sixty-fourth of the codes) a byte that is set
// if it does for all of them.  nvbin is a multiple of 256: a block has a multiple of 4
// codes, and whole words of bits where it has 32 or more
__global__ void __launch_bounds__(1024) k_vdec_build(const float* __restrict__ tan_table, double coef,
                                                    double* __restrict__ out, int nvbin, cube_codec codec, VencTab tab) {
  uint32_t* fix = reinterpret_cast<uint32_t*>(out + nvbin);
  uint8_t* all = reinterpret_cast<uint8_t*>(fix + (nvbin >> 5));
  const int per = nvbin >> 6, c0 = blockIdx.x * per;
  int same_all = 1;
  for (int i = threadIdx.x; i < ((per + 31) & ~31); i += blockDim.x) {  // whole warps
    const int c = c0 + i;
    bool same = true;
    if (i < per) {
      const double v = cube_vdecode(tan_table[c], coef);
      out[c] = v;
      same = cube_wrap_code(cube_vencode_step(&codec, tab, v, coef), codec.izipv) == c - nvbin / 2;
      same_all &= same;
    }
    const uint32_t bits = __ballot_sync(0xffffffffu, same);
    if ((threadIdx.x & 31) == 0 && per >= 32) fix[c >> 5] = bits;
    // fewer codes than a word's: the block's bytes of the word (per = 4: half a byte)
    if (threadIdx.x == 0 && per < 32) {
      atomicAnd(&fix[c >> 5], ~(((1u << per) - 1u) << (c & 31)));
      atomicOr(&fix[c >> 5], (bits & ((1u << per) - 1u)) << (c & 31));
    }
  }
  same_all = __syncthreads_and(same_all);
  if (threadIdx.x == 0) all[blockIdx.x] = (uint8_t)same_all;
}
}  // namespace

// decode table for coef: the velocity decode tan(pi*code/(nvbin-1))/coef of every
// code, computed by the same FP32 table and FP64 division as a per-particle decode,
// so a lookup is bit-identical to it; followed by the bits of cube_vfixed
const double* cube_vdec_table(cube_ctx* ctx, double coef, int* rc) {
  *rc = CUBE_OK;
  for (int i = 0; i < 2; ++i)
    if (ctx->vdec[i] && ctx->vdec_coef[i] == coef) {
      ctx->vdec_next = i ^ 1;  // the caller may ask for another beside it (the kick decodes by two)
      return ctx->vdec[i];
    }
  const int i = ctx->vdec_next;
  ctx->vdec_next ^= 1;
  if (!ctx->vdec[i] && cudaMalloc((void**)&ctx->vdec[i], sizeof(double) * ctx->nvbin + sizeof(uint32_t) * (ctx->nvbin / 32) + 64) !=
                           cudaSuccess) {
    ctx->err = "cudaMalloc of the velocity decode table failed";
    *rc = CUBE_ERR_CUDA;
    return nullptr;
  }
  k_vdec_build<<<64, std::max(32, ctx->nvbin >> 6), 0, ctx->stream>>>(ctx->tan_table, coef, ctx->vdec[i], ctx->nvbin,
                                                                     ctx->codec, cube_venc_tab(ctx));
  ctx->launches++;
  if (cudaGetLastError() != cudaSuccess) {
    ctx->err = "velocity decode table launch failed";
    *rc = CUBE_ERR_CUDA;
    return nullptr;
  }
  ctx->vdec_coef[i] = coef;
  return ctx->vdec[i];
}

namespace {
// velocities spread over the code range: v = tan(pi_f*(code + off)/(nvbin-1))/coef with an
// integer code, so that the encode's q is code + off, and off of a hash of the index: within
// 1.3e-8 of the rounding boundary code + 1/2, within 1e-3 of it (both sides of the edges of the
// FP32 form's band of 2e-4), or anywhere; the step's encode against cube_vencode.
// seen: mismatches, inputs inside the band, inputs beside it
__global__ void k_encode_check(cube_codec codec, VencTab tab, double coef, int64_t n, uint64_t seed,
                               unsigned long long* __restrict__ seen) {
  unsigned long long bad = 0, inside = 0, beside = 0;
  const double nb1 = (double)codec.nvbin_m1_f, pif = (double)codec.pi_f;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    uint64_t h = (uint64_t)i * 0x9E3779B97F4A7C15ull + seed;
    h ^= h >> 31; h *= 0xBF58476D1CE4E5B9ull; h ^= h >> 27; h *= 0x94D049BB133111EBull; h ^= h >> 31;
    const double u = (double)(h >> 19) * 0x1p-45;                     // [0,1), of other bits than cls and off
    const double code = floor(u * (nb1 + 1.0)) - 0.5 * (nb1 + 1.0);   // every code
    const int cls = (int)(h & 7);
    const double off = cls < 3 ? ((double)((h >> 3) & 0xFF) - 128.0) * 1e-10 + 0.5
                     : cls < 6 ? ((double)((h >> 3) & 0xFFFF) - 32768.0) * 3e-8 + 0.5
                               : ((double)((h >> 3) & 0xFFFF) / 65536.0 - 0.5);
    const double ang = pif * (code + off) / nb1;
    if (fabs(ang) >= 1.5707963) continue;
    const double v = tan(ang) / coef;
    const double q = nb1 * atan(coef * v) / pif, d = fabs(q - floor(q) - 0.5);
    inside += d < (double)VENC_BAND;
    beside += d >= (double)VENC_BAND && d < 1e-3;
    bad += cube_vencode_step(&codec, tab, v, coef) != cube_vencode(&codec, v, coef);
  }
  if (bad) atomicAdd(seen, bad);
  atomicAdd(seen + 1, inside);
  atomicAdd(seen + 2, beside);
}
}  // namespace

namespace {
// splitmix64 stream for the division check
__device__ __forceinline__ uint64_t smix(uint64_t& s) {
  uint64_t z = (s += 0x9E3779B97F4A7C15ull);
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}

// quotients of the PP pair term x/r^3 (x a separation component on the 2^-14 or 2^-6
// grid of int2/int1 positions within +-8 fine cells, r^3 from three such components,
// r > 0.3) and of random doubles over wide ranges: cube_div_rcp against __ddiv_rn
__global__ void k_division_check(int64_t n, uint64_t seed, unsigned long long* bad) {
  unsigned long long nb = 0;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    uint64_t st = seed ^ (0xD1B54A32D192ED03ull * (uint64_t)(i + 1));
    const int kind = (int)(i & 3);
    double a[3], b;
    if (kind < 3) {
      const double res = kind == 2 ? 0.015625 : 6.103515625e-05;  // 2^-6 or 2^-14
      const int span = kind == 2 ? 1024 : 262144;                // +-8 fine cells
      double r2 = 0.0;
      for (int d = 0; d < 3; ++d) {
        a[d] = res * (double)((int64_t)(smix(st) % (uint64_t)(2 * span + 1)) - span);
        r2 = __dadd_rn(r2, __dmul_rn(a[d], a[d]));
      }
      const double rm = sqrt(r2);
      if (!(rm > 0.3)) continue;
      b = __dmul_rn(__dmul_rn(rm, rm), rm);
    } else {
      const uint64_t u = smix(st);
      b = ldexp(1.0 + (double)(u >> 12) * 0x1p-52, (int)(smix(st) % 50) - 10);
      for (int d = 0; d < 3; ++d) {
        const uint64_t v = smix(st);
        a[d] = ldexp(1.0 + (double)(v >> 12) * 0x1p-52, (int)(smix(st) % 60) - 30) * ((v & 1) ? -1.0 : 1.0);
      }
    }
    const double y = __drcp_rn(b);
    for (int d = 0; d < 3; ++d) {
      const double q1 = cube_div_rcp(a[d], b, y), q2 = __ddiv_rn(a[d], b);
      if (__double_as_longlong(q1) != __double_as_longlong(q2)) ++nb;
    }
  }
  if (nb) atomicAdd(bad, nb);
}
}  // namespace

int32_t cube_debug_division_check(cube_ctx* ctx, int64_t n, uint64_t seed, int64_t* mismatches) {
  if (!ctx || !mismatches || n < 0) return CUBE_ERR_PARAM;
  unsigned long long* bad = reinterpret_cast<unsigned long long*>(ctx->red_tmp);
  CUBE_CUDA_TRY(ctx, cudaMemsetAsync(bad, 0, 8, ctx->stream));
  k_division_check<<<ctx->num_sms * 8, 256, 0, ctx->stream>>>(n, seed, bad);
  CUBE_LAUNCH_CHECK(ctx);
  unsigned long long h = 0;
  CUBE_CUDA_TRY(ctx, cudaMemcpyAsync(&h, bad, 8, cudaMemcpyDeviceToHost, ctx->stream));
  CUBE_CUDA_TRY(ctx, cudaStreamSynchronize(ctx->stream));
  *mismatches = (int64_t)h;
  return CUBE_OK;
}

int32_t cube_debug_encode_check(cube_ctx* ctx, int64_t n, uint64_t seed, float sigma, int64_t* mismatches) {
  if (!ctx || !mismatches || n < 0) return CUBE_ERR_PARAM;
  unsigned long long* seen = reinterpret_cast<unsigned long long*>(ctx->red_tmp);
  unsigned long long h[3] = {0, 0, 0};
  CUBE_CUDA_TRY(ctx, cudaMemsetAsync(seen, 0, sizeof(h), ctx->stream));
  const double coef = cube_vcoef(&ctx->codec, sigma);
  k_encode_check<<<ctx->num_sms * 8, 256, 0, ctx->stream>>>(ctx->codec, cube_venc_tab(ctx), coef, n, seed, seen);
  CUBE_LAUNCH_CHECK(ctx);
  CUBE_CUDA_TRY(ctx, cudaMemcpyAsync(h, seen, sizeof(h), cudaMemcpyDeviceToHost, ctx->stream));
  CUBE_CUDA_TRY(ctx, cudaStreamSynchronize(ctx->stream));
  *mismatches = (int64_t)h[0];
  // 3/8 and a fifth of another 3/8 of the inputs lie inside the band, the rest of those beside it
  if (n >= 4096 && (h[1] < (unsigned long long)n / 4 || h[2] < (unsigned long long)n / 8)) {
    ctx->err = "encode check: " + std::to_string(h[1]) + " inputs inside the band and " + std::to_string(h[2]) +
               " beside it of " + std::to_string(n);
    return CUBE_ERR_STATE;
  }
  return CUBE_OK;
}
