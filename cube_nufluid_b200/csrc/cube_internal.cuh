/*
 * cube_internal.cuh -- device state and launch helpers of the B200 PM step.
 *
 * Device layout (one image on one GPU; tiles are only an ordering):
 *   cell id   c = ((tz*nnt+ty)*nnt+tx)*nt^3 + (lz*nt+ly)*nt + lx
 *             (Fortran rhoc(lx,ly,lz,tx,ty,tz) order, variables.f90:65)
 *   particles cell-sorted, each particle stored once (no buffer copies);
 *             SoA: xp[d][cap], vp[d][cap] (1 or 2 bytes), pid[cap]
 *   cell_start[c] (int64, exclusive prefix of rhoc), vfield[d][ncells]
 *   fine mesh nf^3 with row pitch rp = nf+32 floats (128-byte rows), used
 *             in place as the half spectrum (complex pitch cp = rp/2)
 *   coarse mesh nc^3, same convention
 */
#ifndef CUBE_INTERNAL_CUH
#define CUBE_INTERNAL_CUH

#include <cuda_runtime.h>
#include <stdint.h>
#include <string.h>

#include <cmath>
#include <string>
#include <vector>

#include "../../include/cube_gpu.h"
#include "cube_codec.h"

#define CUBE_MAX_RADIX_STAGES 12

struct FftPlan {
  int n;                          // transform length
  int nst;                        // number of stages
  int radix[CUBE_MAX_RADIX_STAGES];
  float2* tw;                     // device twiddles exp(-2 pi i j/n), j < n
  float2* tw2;                    // register-FFT twiddles tw[(t*k1) mod n] at [k1*T + t] (n = R*T)
  double2* twd;                   // tw in FP64 (FP64 Poisson mode)
};

// R x T split of the register-resident transforms (T threads of one warp, R
// points each); false for lengths they do not cover
inline bool cube_fast_rt(int n, int* R, int* T) {
  switch (n) {
    case 1024: *R = 32; *T = 32; return true;
    case 512: *R = 32; *T = 16; return true;
    case 256: *R = 16; *T = 16; return true;
    case 128: *R = 16; *T = 8; return true;
    case 64: *R = 8; *T = 8; return true;
    case 32: *R = 8; *T = 4; return true;
    case 768: *R = 48; *T = 16; return true;
    case 384: *R = 48; *T = 8; return true;
    case 192: *R = 24; *T = 8; return true;
    case 96: *R = 24; *T = 4; return true;
    default: return false;
  }
}

struct MeshLevel {
  int n;          // mesh points per dimension
  int rp;         // real row pitch (floats)
  int cp;         // complex row pitch (float2) = rp/2
  size_t plane;   // floats per z-plane = n*rp
  float* rho;     // density, in place as the forward half spectrum
  float* force;   // [3] force meshes, each n*plane floats, in place as spectra
  float* ext;     // scratch mesh (n*plane floats) for the transposed passes
  float* kern;    // Green multiplier (imaginary parts, /n^3)
  double* kernd = nullptr;  // the same in FP64 (FP64 Poisson mode, else null)
  int fp64 = 0;             // 1: rho, force and ext hold doubles (same element pitches)
  int kern_octant;  // 1: kern is [3][(n/2+1)^3] octant; 0: [3][n][n][cp_k]
  int kern_pitch;   // inner pitch of kern (n/2+1)
  FftPlan plan;
};

struct DevScal {
  unsigned int f2_fine_bits;   // max f^2 as float bits (non-negative floats order as ints)
  unsigned int f2_coarse_bits;
  unsigned int vmax_bits[3];
  unsigned int f2_pp_bits;
  int err;                     // first error code seen on the device
  int err_info;
  unsigned long long n_big;    // re-bin cells for the warp sorter (PP: spilled bricks)
  unsigned long long itest1, npairs;
  unsigned long long moved_far;
  unsigned int nu_dt_bits[3];  // per-fluid CFL step as float bits
  unsigned long long n_huge;   // re-bin cells beyond the shared-memory sorter
  unsigned long long max_huge; // the most particles in one of them
  unsigned long long n_mid;    // re-bin cells for the block sorter (beyond the warp sorter)
  unsigned long long huge_next;  // next cell for a k_rebin_huge block
  unsigned long long n_items;    // re-bin work items beyond the one per 64-cell group
  unsigned long long mid_next;   // next cell for a k_rebin_big block
  unsigned long long n_dep_extra;  // deposit work items beyond one per brick
  unsigned long long n_split;      // bricks whose particles are split over several deposit blocks
  unsigned long long pp_list;      // PP targets with a neighbour, listed for the pair pass
  unsigned long long pp_dense;     // PP bricks whose region holds a crowded cell
  unsigned int kick_next;          // next work item for a group of k_kick_p
  unsigned long long mass[3];      // deposit: fine and coarse particle sums, coarse neutrino sum (fixed point)
  long long np_new;                // particles the re-bin counted
  double sums[3];                  // tree sums: |vfield|^2, |v_res|^2, |v|^2 (particle mesh: [0] fine neutrino mass)
};

// one isothermal fluid of the dispersive sum (hydrogr.f90 type hydro): five FP32
// arrays of n^3 cells, x fastest, periodic; a = current state, b = the other
// half of the ping-pong (each is one contiguous block of 5 n^3)
struct NuFluid {
  int n = 0, ncb = 0;              // cells per side; halo width of the reference layout
  float dx = 0.f, cs2 = 0.f, dv = 0.f;
  float* a[5] = {nullptr, nullptr, nullptr, nullptr, nullptr};
  float* b[5] = {nullptr, nullptr, nullptr, nullptr, nullptr};
  float* block[2] = {nullptr, nullptr};
  float* xy = nullptr;             // gravity scratch [5][nf+4][n][n]
};

// fluid neutrinos of one species (hydrodf.f90 type dfld)
struct NuState {
  bool on = false;
  float beta = 0.f, g = 0.f, ai = 0.f;
  float dwgts[3] = {0.f, 0.f, 0.f};
  NuFluid fl[3];
  double* partial = nullptr;       // per-CTA sums of the fine neutrino density
  int nparts = 0;
};

// the calls that are timed (cube_phase_times)
enum EvCall { EV_UPDATE_X, EV_PP, EV_PARTICLE_MESH, EV_NU };

struct cube_ctx {
  cube_params P;
  int nc, nnt, nt, ncell, ncb, nte, nf, nvbin;
  int64_t ncells;
  int izipx, izipv;
  cube_codec codec;
  cudaStream_t stream;
  cudaStream_t side = nullptr;                      // beside it, for the re-bin of the largest cells (made on
  cudaEvent_t side_ev[2] = {nullptr, nullptr};      // first use); it begins after and ends before work of stream
  int own_stream;
  int64_t np, cap;
  int state_loaded;
  int cells_le32;  // the last re-bin left no cell beyond 32 particles (no deposit brick needs splitting)
  int num_sms;
  // particles (double-buffered for the re-bin)
  void* xp;  void* vp;  int32_t* pid;
  void* xp2; void* vp2; int32_t* pid2;
  int32_t* rhoc;  int32_t* rhoc2;
  int64_t* cell_start; int64_t* cell_start2;
  float* vfield; float* vfield2;
  // re-bin scratch
  int32_t* tcell; uint32_t* tkey; int32_t* perm; uint32_t* pkey; int32_t* cursor;
  int32_t* big_list;
  int64_t* rebin_items;  // [4] per item: first cell, cells, first and end particle
  double* cell_stats;   // [3][ncells]
  double* slot_r2; double* slot_s2;  // re-bin scratch: each slot's new cell (int32), tree block sums
  double* red_tmp;      // scratch for tree sums
  int64_t* scan_tmp;
  NuState nu;
  double* pk_bins;  // power-spectrum bin sums, 7 * (bins of the fine mesh + 1)
  double* vdec[2] = {nullptr, nullptr};  // decoded velocity per code, tan(code)/coef, for two coefs
  double vdec_coef[2] = {0.0, 0.0};
  int vdec_next = 0;
  void* pp_scratch = nullptr;     // sorted particles of crowded PP bricks, grown on demand
  size_t pp_scratch_bytes = 0;
  void* rebin_scratch = nullptr;  // sort slots of re-bin cells beyond 4096 particles, grown on demand
  size_t rebin_scratch_bytes = 0;
  void* rebin_mid_scratch = nullptr;  // velocity columns of the block sorter, allocated on first use
  void* dep_scratch = nullptr;   // fine nodes and block counters of split deposit bricks, grown on demand
  size_t dep_scratch_bytes = 0;
  void* halo_shells = nullptr;   // the halo finder's list of cell offsets by distance, made on first use
  // meshes
  MeshLevel fine, coarse;
  unsigned long long* rho_c_acc;  // coarse particle sums, 64-bit fixed point without the mass (scale 2^38)
  unsigned long long* rho_c_nu;   // coarse neutrino sums, 64-bit fixed point in mass units (scale 2^32)
  double* dep_partial;            // per-CTA fine mass partial sums
  int64_t dep_blocks;
  float* tan_table;               // tanf of each velocity code, index code+nvbin/2
  int tan_odd;                    // 1: tan_table[half - k] = -tan_table[half + k] for every k, bit for bit
  struct VencBrk* venc_brk;       // breakpoints of cube_vencode_step (VENC_N entries)
  DevScal* dscal;                 // device scalars
  DevScal* hscal;                 // pinned host mirror
  float2* sbuf;                   // spare spectrum buffer for the forward z pass
  // timing
  // events of the calls that are timed, twice: a call records into the set that its last
  // finished one did not use, so that one which fails leaves the times that are there
  cudaEvent_t ev[2][16] = {};
  int ev_set[4] = {0, 0, 0, 0};     // the set that each call (EvCall) records into next
  cudaEvent_t phase_ev[8][2] = {};  // first and last event of each phase of the last finished calls
  std::vector<const void*> smem_raised;  // kernels whose dynamic shared-memory limit this context has raised
  long long launches;
  std::string err;
};

// ---- error helpers ---------------------------------------------------------
#define CUBE_CUDA_TRY(ctx, call)                                                   \
  do {                                                                             \
    cudaError_t e_ = (call);                                                       \
    if (e_ != cudaSuccess) {                                                       \
      (ctx)->err = std::string(#call) + ": " + cudaGetErrorString(e_);             \
      return CUBE_ERR_CUDA;                                                        \
    }                                                                              \
  } while (0)

#define CUBE_LAUNCH_CHECK(ctx)                                                     \
  do {                                                                             \
    (ctx)->launches++;                                                             \
    cudaError_t e_ = cudaGetLastError();                                           \
    if (e_ != cudaSuccess) {                                                       \
      (ctx)->err = std::string("launch: ") + cudaGetErrorString(e_);               \
      return CUBE_ERR_CUDA;                                                        \
    }                                                                              \
  } while (0)

__device__ __forceinline__ void cube_dev_error(DevScal* s, int code, int info) {
  if (atomicCAS(&s->err, 0, code) == 0) s->err_info = info;
}

// Raises a kernel's dynamic shared-memory limit to the most the device allows beside
// the kernel's static shared memory, on the context's first launch of it (the calls
// lock the driver: with several contexts on as many threads they took longer than
// the kernels of a small box).  The limit is a per-kernel global, so contexts on other
// host threads launching the same kernel with other sizes must never see it lowered
// under them: it is only ever set to that one value.  A launch that needs more fails.
template <typename F>
inline cudaError_t cube_smem_limit(cube_ctx* ctx, F* func, size_t bytes) {
  if (bytes == 0) return cudaSuccess;
  const void* key = reinterpret_cast<const void*>(func);
  for (const void* k : ctx->smem_raised)
    if (k == key) return cudaSuccess;
  int dev = 0, optin = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  cudaFuncAttributes fa;
  if (e == cudaSuccess) e = cudaFuncGetAttributes(&fa, func);
  if (e != cudaSuccess) return e;
  const size_t lim = (size_t)optin > fa.sharedSizeBytes ? (size_t)optin - fa.sharedSizeBytes : 0;
  if (bytes > lim) return cudaErrorInvalidValue;
  e = cudaFuncSetAttribute(func, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)lim);
  if (e == cudaSuccess) ctx->smem_raised.push_back(key);
  return e;
}

// sum of v over the block (a multiple of 32 threads, at most 1024), valid in thread 0;
// every thread calls it
__device__ __forceinline__ unsigned long long cube_block_sum(unsigned long long v) {
  __shared__ unsigned long long ws[32];
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = v;
  __syncthreads();
  unsigned long long t = 0ull;
  if (threadIdx.x == 0)
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += ws[w];
  __syncthreads();
  return t;
}
// maximum of v over the block, valid in thread 0
__device__ __forceinline__ unsigned int cube_block_max(unsigned int v) {
  __shared__ unsigned int wm[32];
  v = __reduce_max_sync(0xffffffffu, v);
  if ((threadIdx.x & 31) == 0) wm[threadIdx.x >> 5] = v;
  __syncthreads();
  unsigned int t = 0u;
  if (threadIdx.x == 0)
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t = max(t, wm[w]);
  __syncthreads();
  return t;
}

// device-side view of the particle codes
template <int Z>
struct CodeT;
template <>
struct CodeT<1> { typedef int8_t T; };
template <>
struct CodeT<2> { typedef int16_t T; };

__device__ __forceinline__ int64_t cube_cell_of(int gx, int gy, int gz, int nt, int nnt) {
  const int tx = gx / nt, ty = gy / nt, tz = gz / nt;
  const int lx = gx - tx * nt, ly = gy - ty * nt, lz = gz - tz * nt;
  return ((((int64_t)tz * nnt + ty) * nnt + tx) * nt + lz) * (int64_t)nt * nt + (int64_t)ly * nt + lx;
}

// n/d for n < 2^31 by a multiply and a shift: with 2^(l-1) < d <= 2^l and
// m = floor(2^(31+l)/d) + 1, n m 2^-(31+l) exceeds n/d by less than 1/d.  m = 0 marks
// a divisor (1) or a use (dividends of 2^31 and more) that takes the division itself.
struct FastDiv {
  uint32_t d, m, s;
};
inline FastDiv cube_fastdiv(uint32_t d, bool wide = false) {
  FastDiv f = {d, 0u, 0u};
  if (d > 1 && !wide) {
    uint32_t l = 1;
    while (((uint64_t)1 << l) < d) ++l;
    f.m = (uint32_t)(((uint64_t)1 << (31 + l)) / d + 1);
    f.s = l - 1;
  }
  return f;
}
__device__ __forceinline__ uint32_t operator/(uint32_t n, const FastDiv& f) {
  return f.m ? __umulhi(n, f.m) >> f.s : n / f.d;
}

// periodic wrap of an index that lies in [-n, 2n)
__device__ __forceinline__ int cube_wrap(int x, int n) {
  x += (x < 0) ? n : 0;
  return x - ((x >= n) ? n : 0);
}

// tile-major cell id -> coordinates inside its tile (l) and the tile's first
// global coarse cell per dimension (tb = tile index * nt)
__device__ __forceinline__ void cube_cell_coords(int64_t c, int nt, int nnt, int l[3], int tb[3]) {
  const int nt3 = nt * nt * nt;
  const int64_t tile = c / nt3;
  const int rem = (int)(c - tile * nt3);
  const int t2 = (int)tile;  // < nnt^3 < 2^31
  l[0] = rem % nt;
  l[1] = (rem / nt) % nt;
  l[2] = rem / (nt * nt);
  tb[0] = (t2 % nnt) * nt;
  tb[1] = ((t2 / nnt) % nnt) * nt;
  tb[2] = (t2 / (nnt * nnt)) * nt;
}

// The kick chain of the reference, (((f*a_mid)*dt)/6)/pi (pm.f90:146,163,358,393),
// is the same for every particle that reads a force node.  cube_particle_mesh folds
// the scalar ((a_mid*dt)/6)/pi into the Green multiply, so the force meshes come
// out of the inverse FFT as kick increments (to FP32 rounding, like the force
// itself); forces given from outside (cube_debug_kick_with_force) get the exact
// per-node chain below.
struct KickScale {
  float a_mid, dt, pi_f;
  int on;
  float inv6, inv_pi;  // RN(1/6), RN(1/pi_f)
};

// RN(x/y) for a constant y with z = RN(1/y): q0 = RN(x z), r = fma(-q0, y, x),
// q = fma(r, z, q0) (Brisebarre, Muller and Raina, IEEE Trans. Computers 53(8),
// 2004).  For y = 6 and y = pi_f the result equals IEEE division for every finite
// FP32 x with |x| >= 2^-100 (checked over all 2^32 inputs by the CPU tests); smaller
// and non-finite x take the IEEE division.
__device__ __forceinline__ float cube_div_const(float x, float y, float z) {
  const float ax = fabsf(x);
  if (!(ax >= 7.88860905e-31f && ax <= 3.40282347e38f)) return __fdiv_rn(x, y);
  const float q0 = __fmul_rn(x, z);
  const float r = __fmaf_rn(-q0, y, x);
  return __fmaf_rn(r, z, q0);
}

// RN(a/b) from y = RN(1/b) for b > 0 (normal) and finite a, by two FMA corrections
// of q0 = RN(a y): the first gives a quotient within one ulp of a/b, and then, y being
// within half an ulp of 1/b, RN(q + (a - b q) y) with the exact FMA residual is the
// correctly rounded quotient (Markstein's theorem; Markstein, IBM J. Res. Dev. 34(1),
// 1990; Muller et al., Handbook of Floating-Point Arithmetic, sec. 4.7).  It replaces
// IEEE divisions by one b shared by several a; cube_debug_division_check compares it
// with the IEEE division on the GPU.
__device__ __forceinline__ double cube_div_rcp(double a, double b, double y) {
  double q = __dmul_rn(a, y);
  double r = __fma_rn(-b, q, a);
  q = __fma_rn(r, y, q);
  r = __fma_rn(-b, q, a);
  return __fma_rn(r, y, q);
}

// The tangents of the codes 0 .. half in shared memory (half + 1 floats; tan is odd), loaded
// by the whole block; and the tangent of a code from them.  A kernel that decodes many
// scattered codes and keeps its CTAs on the SM reads 32 codes of a warp from them in three or four
// cycles, and forms the decode table's entry by cube_div_rcp; in the tables (half a
// megabyte each) they are 32 lines.  From CUBE_TAN_MIN particles the loads of the tangents
// are small beside the kernels' time (the figures of both sides stand at the launches).
constexpr int64_t CUBE_TAN_MIN = 1 << 19;
// The quotient through the reciprocal is the IEEE one for ordinary coefficients only: an
// infinite one (a velocity dispersion of zero) gives 0 in the tables and NaN there.
inline bool cube_use_tan(const cube_ctx* ctx, double coef) {
  return ctx->np >= CUBE_TAN_MIN && ctx->tan_odd && coef > 1e-100 && coef < 1e100;
}
__device__ __forceinline__ void cube_tan_load(float* tan_s, const float* __restrict__ tan_table, int half) {
  for (int i = threadIdx.x; i < half; i += blockDim.x) tan_s[i] = tan_table[half + i];
  if (threadIdx.x == 0) tan_s[half] = -tan_table[0];  // code -half alone has this magnitude
}
__device__ __forceinline__ double cube_tan_of(const float* tan_s, int code) {
  return (double)__int_as_float(__float_as_int(tan_s[abs(code)]) ^ (code & 0x80000000));
}

inline float cube_kick_scalar(const KickScale& k) {
  return k.on ? cube_fdiv(cube_fdiv(cube_fmul(k.a_mid, k.dt), 6.f), k.pi_f) : 1.f;
}

__device__ __forceinline__ float cube_kick_scale(float f, const KickScale& k) {
  const float t = __fmul_rn(__fmul_rn(f, k.a_mid), k.dt);
  return cube_div_const(cube_div_const(t, 6.f, k.inv6), k.pi_f, k.inv_pi);
}

// Velocity encode in FP32 with a certified rounding.  The code is the integer nearest
// to q = Q atan(x), x = coef v, Q = nvbin_m1/pi_f, so FP32 arithmetic decides it unless
// q lies close to k + 1/2.  x is split off the nearest of the VENC_N breakpoints c_j
// (32 per octave from 2^-7 to 2^9, found from the bits of the FP32 x; c_0 = 0 below
// 2^-7): atan(x) = atan(c_j) + atan(u), u = (x - c_j)/(1 + x c_j), |u| <= 2^-7 (just below 2^-7,
// where c_0 = 0, and nearly so above 1), and Q atan(c_j) is tabulated as an integer plus an FP32
// rest.  The difference x - c_j is formed in FP64 (c_j has seven significant bits, so the
// high word of its double is all of it) and rounded once.  Q atan(u) reaches 163 in magnitude.
// Its relative error, in units of 2^-24: 1 from the difference, 2 from the denominator, 4 from
// the approximate quotient (2 ulp), 1.5 from the polynomial, 1 from Q; in all 9.3e-5 at 163, and
// 8e-6 from the final multiply-add and 2e-7 from the dropped u^5/5 (at most 6e-12) beside it: at
// most 1.02e-4 where everything falls together.  The integer is accepted unless the fraction comes
// within VENC_BAND = 2e-4 of 1/2, twice that (one encode in 2500), where the exact FP64
// evaluation decides, as it does beyond 2^9 and for NaN.  (An FP64 evaluation from 64 angle
// breakpoints with a 1e-9 band, the form before, took 83 warp instructions per encode and six
// conversions; this takes 30.)
constexpr int VENC_LO = 120, VENC_OCT = 16;        // first octave 2^(120-127), octaves
constexpr int VENC_N = VENC_OCT * 32 + 1;
constexpr float VENC_BAND = 2e-4f;
struct VencBrk {
  uint32_t c_hi;  // high word of c_j as a double (its low word is zero)
  float c;        // the same as a float
  int32_t n;      // Q atan(c_j) = n + f, |f| <= 1/2
  float f;
};
struct VencTab {
  const VencBrk* brk;  // VENC_N breakpoints
  float q;             // Q
};
inline VencTab cube_venc_tab(const cube_ctx* ctx) {
  return VencTab{ctx->venc_brk, (float)((double)ctx->codec.nvbin_m1_f / (double)ctx->codec.pi_f)};
}

// the breakpoint table of a codec, on the host
inline std::vector<VencBrk> cube_venc_breakpoints(const cube_codec& codec) {
  std::vector<VencBrk> t(VENC_N);
  const long double Q = (long double)codec.nvbin_m1_f / (long double)codec.pi_f;
  for (int j = 0; j < VENC_N; ++j) {
    // the middle of the floats whose bits >> 18 are (VENC_LO << 5) + j - 1
    const double c = j ? ldexp(1.0 + ((j - 1) % 32 + 0.5) / 32.0, VENC_LO - 127 + (j - 1) / 32) : 0.0;
    uint64_t b;
    memcpy(&b, &c, 8);
    const long double q = Q * atanl((long double)c);
    t[j].c_hi = (uint32_t)(b >> 32);
    t[j].c = (float)c;
    t[j].n = (int32_t)llroundl(q);
    t[j].f = (float)(q - (long double)t[j].n);
  }
  return t;
}

// the encode of the step's kernels (kick, PP, re-bin, decode-table fixed points)
__device__ __forceinline__ int32_t cube_vencode_step(const cube_codec* c, const VencTab& T, double v, double coef) {
  const double x = cube_dmul(coef, v);
  const double ax = fabs(x);
  const float xf = __double2float_rn(ax);
  const uint32_t b = __float_as_uint(xf);
  if (!(xf < 512.f)) return cube_vencode(c, v, coef);  // beyond the table, or NaN
  const int j = max((int)(b >> 18) - ((VENC_LO << 5) - 1), 0);
  const uint4 e = __ldg(reinterpret_cast<const uint4*>(T.brk + j));
  const float num = __double2float_rn(cube_dsub(ax, __hiloint2double((int)e.x, 0)));
  const float u = __fdividef(num, __fmaf_rn(xf, __uint_as_float(e.y), 1.f));
  const float p = __fmul_rn(u, __fmaf_rn(__fmul_rn(u, u), -0.333333343f, 1.f));  // atan(u)
  const float t = __fmaf_rn(T.q, p, __uint_as_float(e.w));
  const float r = rintf(t);
  if (fabsf(__fsub_rn(t, r)) > 0.5f - VENC_BAND) return cube_vencode(c, v, coef);
  const int32_t n = (int32_t)e.z + (int)r;  // >= 0
  return x < 0.0 ? -n : n;
}

// ---- launchers (implemented in the k_*.cu files) -----------------------------
// drift and re-bin into the second buffers.  Without `crowded`, everything but the cells
// of more than 32 particles, whose counts are left in DevScal; with it (after a look at
// those counts) the crowded cells alone.
int cube_rebin(cube_ctx* ctx, cube_scalars* io, bool crowded);
inline bool cube_rebin_has_crowded(const cube_ctx* ctx) {
  return (ctx->hscal->n_big | ctx->hscal->n_mid | ctx->hscal->n_huge) != 0ull;
}
// DevScal into its pinned mirror, and the stream finished
inline cudaError_t cube_read_dscal(cube_ctx* ctx) {
  cudaError_t e = cudaMemcpyAsync(ctx->hscal, ctx->dscal, sizeof(DevScal), cudaMemcpyDeviceToHost, ctx->stream);
  return e == cudaSuccess ? cudaStreamSynchronize(ctx->stream) : e;
}
int64_t cube_rebin_items_max(int64_t ncells, int64_t cap);
// Work items over the cells of cell_start (a run of at most 64 cells and at most 4096 of
// its particles each); *blocks = launch size, one block per item, blocks past the last
// return (cube_cell_item).  Returned in ctx->rebin_items, or null when every cell is
// known to hold at most 32 particles: a group of 64 cells is then an item, read
// from the cell starts without a list (two launches of a small box's step saved twice,
// and a third of a large box's blocks, which found nothing to do).
int cube_cell_items(cube_ctx* ctx, const int64_t* cell_start, bool le32, const int64_t** items, int64_t* blocks);
__device__ __forceinline__ bool cube_cell_item(const int64_t* items, int64_t ncells, int64_t items_max,
                                               const DevScal* dscal, const int64_t* cell_start, int64_t b,
                                               int64_t& c0, int& ncl, int64_t& p0, int64_t& p1) {
  const int64_t ngroups = (ncells + 63) / 64;
  if (!items) {
    if (b >= ngroups) return false;
    c0 = b * 64;
    ncl = (int)min((int64_t)64, ncells - c0);
    p0 = cell_start[c0];
    p1 = cell_start[c0 + ncl];
    return true;
  }
  if (b >= ngroups + (int64_t)dscal->n_items || b >= items_max) return false;
  const int64_t* it = items + 4 * b;
  c0 = it[0]; ncl = (int)it[1]; p0 = it[2]; p1 = it[3];
  return true;
}
int cube_deposit(cube_ctx* ctx, cube_scalars* io);
// mass sums of a deposit (pm.f90:108,280) from the three totals it leaves in
// DevScal::mass: fine and coarse particle sums without the mass (scale 2^32) and
// the coarse neutrino sum (mass units, scale 2^32); the caller adds the fine
// neutrino sum
inline void cube_mass_sums(const unsigned long long mt[3], float mass, double* testrhof, double* testrhoc) {
  const double m = (double)mass, s = 1.0 / 4294967296.0;
  *testrhof = (double)mt[0] * s * m;
  *testrhoc = (double)mt[1] * s * m + (double)mt[2] * s;
}
int cube_fft_poisson(cube_ctx* ctx, MeshLevel& L, unsigned int* f2_bits, KickScale ks);
int cube_force_scale(cube_ctx* ctx, MeshLevel& L, KickScale ks);
int cube_fft_forward3(cube_ctx* ctx, MeshLevel& L, float* data, int* kx_major);
int cube_pk_nbin(int ng, int logbins);
int cube_power_spectrum_dev(cube_ctx* ctx, int logbins, std::vector<double>& bins, int* nbin_out);
// compile-time mixed-radix passes (k_fftm.cu) of one mesh size; null if not compiled
struct FftmOps {
  int (*x_r2c)(cube_ctx*, MeshLevel&, float* data);
  int (*x_c2r3)(cube_ctx*, MeshLevel&, float* data, unsigned int* f2_bits);
  int (*col)(cube_ctx*, MeshLevel&, float* data, int ncomp, int along_z, float sgn);
  int (*z_green)(cube_ctx*, MeshLevel&, const float* rho, float* force, const float* kern, float ksc);
};
const FftmOps* cube_fftm_ops(int n);
int cube_fft_forward3_fast(cube_ctx* ctx, MeshLevel& L, float* data, int* rc, int* kx_major);
int cube_fft_poisson_fast(cube_ctx* ctx, MeshLevel& L, unsigned int* f2_bits, KickScale ks, int* rc);
int cube_kick(cube_ctx* ctx, cube_scalars* io);
// *read: the call ended with cube_read_dscal and nothing launched after it
int cube_pp(cube_ctx* ctx, cube_scalars* io, bool* read);
int cube_build_green(cube_ctx* ctx, const float* fk_table, const float* ck_table);
int cube_tree_sum_dev(cube_ctx* ctx, const double* in, int64_t n, double* out_host);
// the same for `count` arrays of n values, `stride` apart, into out_dev[0 .. count-1] on the
// device, without waiting
int cube_tree_sums_async(cube_ctx* ctx, const double* in, int64_t n, int64_t stride, int count, double* out_dev);
// the velocity statistics of update_x in the re-bin's new layout (second buffers), into
// DevScal::sums: sum |vfield|^2 over the cells, sum |v_res|^2 and sum |v|^2 over the
// particles from their codes, their cell means and each slot's cell (slot_cell); dec is
// the decode table of coef
int cube_stats_sums(cube_ctx* ctx, const int32_t* slot_cell, const double* dec, double coef);
// total: also to *total on the device; zero: n counters to clear on the way (both may be null)
int cube_exclusive_scan(cube_ctx* ctx, const int32_t* in, int64_t n, int64_t* out, long long* total = nullptr,
                        int32_t* zero = nullptr);
int cube_fft_plan(cube_ctx* ctx, FftPlan& p, int n);
int cube_nu_init(cube_ctx* ctx, NuFluid& F);
int cube_nu_sweeps(cube_ctx* ctx, NuFluid& F, float dt, int dir);
int cube_nu_timestep(cube_ctx* ctx, NuFluid& F, unsigned int* dt_bits);
int cube_nu_transpose(cube_ctx* ctx, NuFluid& F, int to_soa);
int cube_nu_density(cube_ctx* ctx, cube_scalars* io);
int cube_nu_gravity(cube_ctx* ctx, cube_scalars* io);
int cube_fft_r2c_x(cube_ctx* ctx, MeshLevel& L, float* data, int inverse, int ncomp, unsigned int* f2_bits);
int cube_make_ic_dev(cube_ctx* ctx, const cube_ic_params* icp, cube_scalars* io);
int cube_halofind_dev(cube_ctx* ctx, const cube_scalars* io, const cube_halo_args* ha, cube_halo_result* res);
// device table of cube_vdecode(tan_table[c], coef) for every code c (index code + nvbin/2),
// built on first use of a coefficient; the last two coefficients asked for stay cached, so
// the two of a kick are valid together.  After the nvbin doubles follow nvbin/32 words of
// cube_vfixed bits and 64 bytes, the k-th of them 1 if all codes of the k-th sixty-fourth of
// the range are fixed.
const double* cube_vdec_table(cube_ctx* ctx, double coef, int* rc);

// true if re-encoding the decoded velocity of code index c (code + nvbin/2) at the
// table's coefficient, cube_wrap_code(cube_vencode_step(v)), gives the code back: a
// velocity kicked by exactly zero then keeps its code
__device__ __forceinline__ bool cube_vfixed(const double* dec, int nvbin, int c) {
  return (reinterpret_cast<const uint32_t*>(dec + nvbin)[c >> 5] >> (c & 31)) & 1u;
}

// those bytes as the bits of a word, by a whole warp
__device__ __forceinline__ unsigned long long cube_vfixed_summary(const double* dec, int nvbin) {
  const uint8_t* all =
      reinterpret_cast<const uint8_t*>(reinterpret_cast<const uint32_t*>(dec + nvbin) + (nvbin >> 5)) + (threadIdx.x & 31);
  const unsigned lo = __ballot_sync(0xffffffffu, all[0]), hi = __ballot_sync(0xffffffffu, all[32]);
  return (unsigned long long)hi << 32 | lo;
}

#endif
