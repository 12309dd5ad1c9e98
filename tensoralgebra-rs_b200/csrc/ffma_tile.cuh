// Tiles of a plain f32 or c32 contraction by FFMA, straight from the operands: what the
// tensor-core kernels fall back to for outputs that BF16 planes cannot carry (split_guard
// in device_common.cuh). Operands through a cp.async ring of KS depths per stage, TM x TN
// outputs a thread, sums restarted every 16 k as in the direct tiles. A warp covers 8 TM
// rows and 4 TN columns, so that its operand reads are one or two wavefronts each.
#pragma once

#include "device_common.cuh"

namespace tprims {
namespace dev {

template <bool CPLX, int WARPS_M, int WARPS_N, int TM_, int TN_, int KS_, int STAGES_>
struct FfmaTile {
  using T = typename Elem<float, CPLX>::type;
  static constexpr int E = CPLX ? 2 : 1, TM = TM_, TN = TN_, KS = KS_, STAGES = STAGES_;
  static constexpr int THREADS = 32 * WARPS_M * WARPS_N, BM = WARPS_M * 8 * TM, BN = WARPS_N * 4 * TN;
  static constexpr int VM = TM < 4 ? TM : 4, VN = TN < 4 ? TN : 4;  // neighbouring rows, columns of a thread
  static constexpr int LDA = BM + 4 / E, LDB = BN + 4 / E;          // elements
  static constexpr int A_BYTES = KS * LDA * 4 * E, STAGE = A_BYTES + KS * LDB * 4 * E, BYTES = STAGES * STAGE;
  static_assert(KS % 16 == 0 && STAGE % 16 == 0 && A_BYTES % 16 == 0, "whole restarts, aligned stages");
  static_assert(TM % VM == 0 && TN % VN == 0 && (VM * E) % 4 == 0 && (VN * E) % 4 == 0, "16-byte reads");
  static_assert(THREADS % BM == 0 && THREADS % BN == 0 && THREADS % KS == 0, "a thread keeps its row or depth");

  float re[TM][TN], im[CPLX ? TM : 1][CPLX ? TN : 1];

  // The tile's row (column) of a thread's i-th (j-th) output.
  __device__ static __forceinline__ int row(int tid, int i) {
    return tid / 32 % WARPS_M * 8 * TM + i / VM * 8 * VM + (tid & 7) * VM + i % VM;
  }
  __device__ static __forceinline__ int col(int tid, int j) {
    return tid / 32 / WARPS_M * 4 * TN + j / VN * 4 * VN + (tid >> 3 & 3) * VN + j % VN;
  }

  // One operand's depths [k0, k0 + KS) into [k][row], zero past K; rows past the end
  // repeat the last one.
  template <int B, int LD>
  __device__ static __forceinline__ void gather(T* dst, const T* X, const int64_t* rows, const int64_t* ks, int64_t ld,
                                                int kfast, int64_t r0, int64_t nrows, int64_t k0, int64_t K, int tid) {
    const auto copy = [&](int r, int k, int64_t ro, int64_t ko) {
      const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst + k * LD + r);
      asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;" ::"r"(d), "l"(X + ro + ko), "n"(sizeof(T)),
                   "r"(k0 + k < K ? (int)sizeof(T) : 0)
                   : "memory");
    };
    const auto row_of = [&](int r) {
      const int64_t x = r0 + r < nrows ? r0 + r : nrows - 1;
      return ld ? x : rows[x];
    };
    const auto k_of = [&](int k) {
      const int64_t x = k0 + k < K ? k0 + k : K - 1;
      return ld ? x * ld : ks[x];
    };
    // The offsets first, all at once: a copy keeps later loads behind it.
    constexpr int N = B * KS / THREADS;
    int64_t off[N];
    if (kfast) {
      const int k = tid % KS;
      const int64_t ko = k_of(k);
#pragma unroll
      for (int i = 0; i < N; ++i) off[i] = row_of(tid / KS + i * (THREADS / KS));
#pragma unroll
      for (int i = 0; i < N; ++i) copy(tid / KS + i * (THREADS / KS), k, off[i], ko);
    } else {
      const int r = tid % B;
      const int64_t ro = row_of(r);
#pragma unroll
      for (int i = 0; i < N; ++i) off[i] = k_of(tid / B + i * (THREADS / B));
#pragma unroll
      for (int i = 0; i < N; ++i) copy(r, tid / B + i * (THREADS / B), ro, off[i]);
    }
  }

  // Outputs of the tile at row m0 and column n0 of batch entry h; operands in device
  // memory at their natural alignment; `sync` joins the tile's threads.
  template <class Sync>
  __device__ __forceinline__ void run(const GemmArgs& g, int64_t h, int64_t m0, int64_t n0, char* smem, int tid, Sync&& sync) {
    const int64_t ns = (g.K + KS - 1) / KS;
    const T* A = static_cast<const T*>(g.A) + (g.a_ld ? h * g.K * g.a_ld : g.s.h_a[h]);
    const T* B = static_cast<const T*>(g.B) + (g.b_ld ? h * g.K * g.b_ld : g.s.h_b[h]);
    const auto issue = [&](int64_t s) {
      if (s < ns) {
        char* st = smem + s % STAGES * STAGE;
        gather<BM, LDA>(reinterpret_cast<T*>(st), A, g.s.a_m, g.s.a_k, g.a_ld, g.a_kfast, m0, g.M, s * KS, g.K, tid);
        gather<BN, LDB>(reinterpret_cast<T*>(st + A_BYTES), B, g.s.b_n, g.s.b_k, g.b_ld, g.b_kfast, n0, g.N, s * KS, g.K, tid);
      }
      asm volatile("cp.async.commit_group;" ::: "memory");
    };
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
      for (int j = 0; j < TN; ++j) {
        re[i][j] = 0.f;
        if constexpr (CPLX) im[i][j] = 0.f;
      }
    sync();  // the ring is free
    for (int s = 0; s < STAGES - 1; ++s) issue(s);
    const float sa = CPLX && g.conj_a ? -1.f : 1.f, sb = CPLX && g.conj_b ? -1.f : 1.f;
    const int ar = row(tid, 0) * E, bc = col(tid, 0) * E;
#pragma unroll 1
    for (int64_t s = 0; s < ns; ++s) {
      asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2) : "memory");
      sync();
      issue(s + STAGES - 1);
      const float* a = reinterpret_cast<const float*>(smem + s % STAGES * STAGE) + ar;
      const float* b = reinterpret_cast<const float*>(smem + s % STAGES * STAGE + A_BYTES) + bc;
#pragma unroll 1
      for (int k16 = 0; k16 < KS; k16 += 16) {
        float cr[TM][TN], ci[CPLX ? TM : 1][CPLX ? TN : 1];
#pragma unroll
        for (int i = 0; i < TM; ++i)
#pragma unroll
          for (int j = 0; j < TN; ++j) {
            cr[i][j] = 0.f;
            if constexpr (CPLX) ci[i][j] = 0.f;
          }
#pragma unroll 4
        for (int k = 0; k < 16; ++k) {
          float x[TM * E], y[TN * E];
          const float *ak = a + (k16 + k) * LDA * E, *bk = b + (k16 + k) * LDB * E;
#pragma unroll
          for (int i = 0; i < TM * E; i += 4)
            *reinterpret_cast<float4*>(x + i) = *reinterpret_cast<const float4*>(ak + i / (VM * E) * 8 * VM * E + i % (VM * E));
#pragma unroll
          for (int j = 0; j < TN * E; j += 4)
            *reinterpret_cast<float4*>(y + j) = *reinterpret_cast<const float4*>(bk + j / (VN * E) * 4 * VN * E + j % (VN * E));
#pragma unroll
          for (int i = 0; i < TM; ++i)
#pragma unroll
            for (int j = 0; j < TN; ++j) {
              if constexpr (CPLX) {
                const float xi = sa * x[2 * i + 1], yi = sb * y[2 * j + 1];
                cr[i][j] = fmaf(x[2 * i], y[2 * j], cr[i][j]);
                cr[i][j] = fmaf(-xi, yi, cr[i][j]);
                ci[i][j] = fmaf(x[2 * i], yi, ci[i][j]);
                ci[i][j] = fmaf(xi, y[2 * j], ci[i][j]);
              } else {
                cr[i][j] = fmaf(x[i], y[j], cr[i][j]);
              }
            }
        }
#pragma unroll
        for (int i = 0; i < TM; ++i)
#pragma unroll
          for (int j = 0; j < TN; ++j) {
            re[i][j] += cr[i][j];
            if constexpr (CPLX) im[i][j] += ci[i][j];
          }
      }
    }
  }
};

}  // namespace dev
}  // namespace tprims
