/*
 * k_fftm.cu -- launchers of the compile-time mixed-radix mesh passes (k_fftm.cuh).
 *
 * Sizes: the multiples of 8 up to 640 with no prime factor above 5 that the register
 * rows of k_fftr.cu do not cover, but for 600 (a coarse mesh of it has a fine mesh of
 * 2400^3 nodes, beyond one GPU).  These are all the other mesh sizes that a box of up to 160
 * coarse cells per side has (its coarse mesh of 8 m cells and its fine mesh of four
 * times that), and larger boxes' coarse meshes.  Other sizes, the FP64 Poisson mode
 * and the stockham_only switch take the passes of k_fft.cu.
 */
#include "k_fftm.cuh"

namespace {

using namespace fftm;

template <int N>
int x_r2c(cube_ctx* ctx, MeshLevel& L, float* data) {
  constexpr size_t smem = sizeof(float2) * Row<N>::BUF * PL<N>::G;
  const int npairs = N * N / 2;
  CUBE_CUDA_TRY(ctx, cube_smem_limit(ctx, k_x_r2c<N>, smem));
  k_x_r2c<N><<<(npairs + Row<N>::C - 1) / Row<N>::C, Row<N>::NT, smem, ctx->stream>>>(data, L.rp, npairs, L.plan.tw,
                                                                                     -1.f);
  CUBE_LAUNCH_CHECK(ctx);
  return CUBE_OK;
}

template <int N>
int x_c2r3(cube_ctx* ctx, MeshLevel& L, float* data, unsigned int* f2_bits) {
  constexpr size_t smem = sizeof(float2) * Row<N>::BUF * (PL<N>::G - 1);
  const int npairs = N * N / 2;
  CUBE_CUDA_TRY(ctx, cube_smem_limit(ctx, k_x_c2r3<N>, smem));
  k_x_c2r3<N><<<(npairs + Row<N>::C - 1) / Row<N>::C, Row<N>::NT, smem, ctx->stream>>>(
      data, (size_t)N * L.plane, L.rp, npairs, L.plan.tw, 1.f, f2_bits);
  CUBE_LAUNCH_CHECK(ctx);
  return CUBE_OK;
}

template <int N>
constexpr unsigned col_blocks() {
  return (unsigned)((N * (N / 2 + 1) + Col<N>::C - 1) / Col<N>::C);
}

template <int N>
int col(cube_ctx* ctx, MeshLevel& L, float* data, int ncomp, int along_z, float sgn) {
  constexpr size_t smem = sizeof(float2) * Col<N>::BUF * (PL<N>::G - 1);
  const long long cp = L.cp, pl = (long long)N * cp;
  CUBE_CUDA_TRY(ctx, cube_smem_limit(ctx, k_col<N>, smem));
  k_col<N><<<dim3(col_blocks<N>(), ncomp), Col<N>::NT, smem, ctx->stream>>>(
      reinterpret_cast<float2*>(data), (size_t)N * L.plane / 2, along_z ? pl : cp, along_z ? cp : pl, L.plan.tw, sgn);
  CUBE_LAUNCH_CHECK(ctx);
  return CUBE_OK;
}

template <int N>
int z_green(cube_ctx* ctx, MeshLevel& L, const float* rho, float* force, const float* kern, float ksc) {
  constexpr size_t smem = PL<N>::G > 1 ? sizeof(float2) * Col<N>::BUF * PL<N>::G : 0;
  const long long cp = L.cp, pl = (long long)N * cp;
  CUBE_CUDA_TRY(ctx, cube_smem_limit(ctx, k_z_green<N>, smem));
  k_z_green<N><<<col_blocks<N>(), Col<N>::NT, smem, ctx->stream>>>(
      reinterpret_cast<const float2*>(rho), reinterpret_cast<float2*>(force), (size_t)N * L.plane / 2, pl, cp,
      L.plan.tw, kern, L.kern_pitch, ksc);
  CUBE_LAUNCH_CHECK(ctx);
  return CUBE_OK;
}

template <int N>
const FftmOps* ops() {
  static const FftmOps o = {x_r2c<N>, x_c2r3<N>, col<N>, z_green<N>};
  return &o;
}

}  // namespace

const FftmOps* cube_fftm_ops(int n) {
  switch (n) {
#define CUBE_FM(n) \
  case n: return ops<n>();
    CUBE_FM(8) CUBE_FM(16) CUBE_FM(24) CUBE_FM(40) CUBE_FM(48) CUBE_FM(72) CUBE_FM(80) CUBE_FM(120)
    CUBE_FM(144) CUBE_FM(160) CUBE_FM(200) CUBE_FM(216) CUBE_FM(240) CUBE_FM(288) CUBE_FM(320)
    CUBE_FM(360) CUBE_FM(400) CUBE_FM(432) CUBE_FM(480) CUBE_FM(576) CUBE_FM(640)
#undef CUBE_FM
    default: return nullptr;
  }
}
