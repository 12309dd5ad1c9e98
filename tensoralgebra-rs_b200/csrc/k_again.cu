// Second pass of the plain f32 and c32 tensor-core kernels: marked parts of their tiles by
// FFMA, straight from the operands. Launched after every such call and nearly always
// without work (a few bytes a CTA to look at); a programmatic launch, so that it is set up
// while the first kernel runs.
#include <type_traits>

#include "ffma_tile.cuh"
#include "tc_common.cuh"

namespace tprims {
namespace dev {

namespace {

// The rows of a tile by 64 (c32: 32) of its columns per CTA.
template <bool CPLX>
using AgainTile = typename std::conditional<CPLX, FfmaTile<true, 2, 4, 4, 2, 16, 3>, FfmaTile<false, 2, 4, 8, 4, 16, 3>>::type;

template <bool CPLX>
__global__ void __launch_bounds__(256, 2)
ffma_again_kernel(const __grid_constant__ GemmArgs g, const unsigned char* __restrict__ flags, int64_t units,
                  int64_t tiles_m, int64_t tiles_n, int tile_n, int grouped) {
  using T = typename Elem<float, CPLX>::type;
  using F = AgainTile<CPLX>;
  extern __shared__ __align__(16) char again_smem[];
  asm volatile("griddepcontrol.wait;" ::: "memory");  // the marks are complete
  __shared__ unsigned char marks[256];
  const int tid = threadIdx.x, subs = tile_n / F::BN;
  int64_t first = blockIdx.x;  // of the next 256 units of this CTA
  int looked = 256;            // of the present ones
  for (;;) {
    // The next marked unit: the four parts along the rows in its half of the columns.
    while (looked < 256 && !marks[looked]) ++looked;
    if (looked == 256) {
      if (first >= units) break;
      const int64_t u = first + (int64_t)tid * gridDim.x;
      const uint32_t all = u < units ? *reinterpret_cast<const volatile unsigned char*>(flags + u / subs) : 0;
      const uint32_t bits = all >> ((int)(u % subs) * F::BN >= tile_n / 2 ? 4 : 0) & 15u;
      first += (int64_t)256 * gridDim.x;
      if (!__syncthreads_or((int)bits)) continue;
      marks[tid] = (unsigned char)bits;
      looked = 0;
      __syncthreads();
      continue;
    }
    const int64_t u = first + (int64_t)(looked - 256) * gridDim.x, t = u / subs;
    const int c0 = (int)(u % subs) * F::BN;
    const uint32_t bits = marks[looked++];
    int64_t h, mt, nt;
    if (grouped) {
      tc::tile_coords(t, tiles_m, tiles_n, h, mt, nt);
    } else {
      nt = t % tiles_n;
      mt = t / tiles_n % tiles_m;
      h = t / tiles_n / tiles_m;
    }
    const int64_t m0 = mt * F::BM, n0 = nt * tile_n + c0;
    if (n0 >= g.N) continue;
    F f;
    f.run(g, h, m0, n0, again_smem, tid, [] { __syncthreads(); });
    T* const Dh = static_cast<T*>(g.D) + g.s.h_d[h];
    const T* const Ch = static_cast<const T*>(g.C) + (g.e.beta_zero ? 0 : g.s.h_c[h]);
#pragma unroll
    for (int i = 0; i < F::TM; ++i)
#pragma unroll
      for (int j = 0; j < F::TN; ++j) {
        const int row = F::row(tid, i);
        const int64_t m = m0 + row, n = n0 + F::col(tid, j);
        if (m >= g.M || n >= g.N || !(bits >> (row * (CPLX ? 2 : 1) / 32) & 1u)) continue;
        epilogue_store<float, CPLX>(g.e, f.re[i][j], CPLX ? f.im[CPLX ? i : 0][CPLX ? j : 0] : 0.f,
                                    Ch + (g.e.beta_zero ? 0 : g.s.c_m[m] + g.s.c_n[n]), Dh + g.s.d_m[m] + g.s.d_n[n]);
      }
  }
}

template <bool CPLX>
cudaError_t run_again(const GemmArgs& g, const unsigned char* flags, int64_t tiles, int64_t tiles_m, int64_t tiles_n,
                      int tile_n, bool grouped, int sms, cudaStream_t st) {
  using F = AgainTile<CPLX>;
  static_assert(F::BM == (CPLX ? 64 : 128) && F::THREADS == 256, "a tile's rows");
  auto kern = ffma_again_kernel<CPLX>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, F::BYTES);
  if (e != cudaSuccess) return e;
  const int64_t units = tiles * (tile_n / F::BN), most = 2 * (int64_t)sms;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(units < most ? units : most));
  cfg.blockDim = dim3(F::THREADS);
  cfg.dynamicSmemBytes = F::BYTES;
  cfg.stream = st;
  cudaLaunchAttribute attr = {};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kern, g, flags, units, tiles_m, tiles_n, tile_n, (int)grouped);
}

}  // namespace

cudaError_t launch_ffma_again(int dtype, const GemmArgs& g, const unsigned char* flags, int64_t tiles, int64_t tiles_m,
                              int64_t tiles_n, int tile_n, bool grouped, int sms, cudaStream_t st) {
  return dtype == 2 ? run_again<true>(g, flags, tiles, tiles_m, tiles_n, tile_n, grouped, sms, st)
                    : run_again<false>(g, flags, tiles, tiles_m, tiles_n, tile_n, grouped, sms, st);
}

}  // namespace dev
}  // namespace tprims
