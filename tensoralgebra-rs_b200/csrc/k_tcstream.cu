// f32 and c32 contractions on the tensor cores without a pack pass.
//
// The FFMA pipe (72 TFLOP/s) bounds plain f32 tiles; BF16 products run 20 times
// faster, and an f32 value is exactly the sum of three BF16 values x0 + x1 + x2 (8
// significant bits each; x1 up to 2^-8 and x2 up to 2^-17 of x). Eight of the nine
// BF16 products are formed, all but x2 y2 (at most 2^-34 of the product). Packing the
// planes through HBM costs 1.5 times the operand's bytes twice, which a short or
// moderate K does not win back, so here the split happens on the way into shared
// memory. One persistent CTA per SM, 128 x 128 tiles, 32-deep stages:
//
//   warps 0-7   epilogue: drain the TMEM accumulators to registers, write back
//               (two warps per 32 rows, each half of the columns).
//   warps 8-23  producers, two sets of eight that take every other block; a warp
//               owns 32 rows of A' (or B'), loads its elements through the scatter
//               vectors to registers while the other set splits, splits them and
//               stores the planes in the tensor core's order (K-major core
//               matrices, no swizzle; the 16-byte step between depth groups keeps
//               the stores free of bank conflicts).
//   warp 24     issues tcgen05.mma, eight products per 16-deep step.
//
// Accumulation. The tensor core truncates each sum it forms, a bias that values of one
// sign do not average out. So the leading products x0 y0 of a step, whose 16 16-bit
// products mostly add up exactly, get an accumulator that starts from zero, and the
// seven cross products (2^-8 of them) one of their own over all of K; the epilogue adds
// the steps in FP32, two at a time, into a running sum that starts again every
// TS_FLUSH blocks of 32. Relative error of 2048^2 f32 products on B200 (FFMA tiles ->
// here), uniform on [-1, 1): K = 64 1.4e-7 -> 0.45e-7, K = 512 1.6e-7 -> 0.7e-7; uniform
// on [0, 1): K = 64 1.15e-7 -> 0.5e-7, K = 512 0.61e-7 -> 0.56e-7; u^8 (one sign, heavy
// tail, where the products of a step do not add up exactly): K = 16 0.59e-7 -> 0.75e-7,
// K = 512 0.68e-7 -> 0.83e-7.
//
// c32 runs as the real product of 2M x N x 2K (rows 2m, 2m + 1 of A' hold [re, -im]
// and [im, re], depths 2k, 2k + 1 of B' re and im): the embedding is a sign flip and
// a swap of the split planes, so a complex element is split once.
//
// Values that BF16 planes cannot carry: the producers track the largest and the
// smallest non-zero magnitude of a tile's operands. With an infinity, a NaN or sums near
// overflow, and where outputs are so small that they may have lost bits to underflow, an
// epilogue warp marks its part of the tile, and a second launch computes the marked parts
// by FFMA straight from the operands (k_again.cu). Inside this kernel that code cost every
// call up to a tenth, whichever role ran it, by the register allocation of the others.
//
// Every wait is bounded (a status bit, then the role ends). No cluster, no multicast.
#include <algorithm>
#include <cmath>
#include <type_traits>

#include "tc_common.cuh"

namespace tprims {
namespace dev {

namespace {

using namespace tc;

constexpr int TS_BM = 128, TS_BN = 128, TS_BK = 32, TS_STAGES = 4;
constexpr int TS_LBO = TS_BM * 16 + 16;     // bytes between 8-deep groups of a plane
constexpr int TS_PLANE = 4 * TS_LBO;        // 128 rows x 32 k
constexpr int TS_STAGE = 6 * TS_PLANE;      // three planes of A', three of B'
constexpr int TS_THREADS = 896;
constexpr int TS_CPT = TS_BN / 2;           // columns of an epilogue warp
constexpr int TS_STATS = 4;                 // tiles whose value ranges are kept
constexpr int TS_FLUSH = 8;                 // 32-deep blocks in a running sum
constexpr int TS_TILES = 15 * 1024;         // tiles of a CTA at most (a byte each)

struct TsSmem {
  static constexpr int RING = TS_STAGES * TS_STAGE;
  static constexpr int COLS = 8 * 4 * TS_CPT * 8;  // per epilogue warp: d_n, c_n of two tiles
  static constexpr int STAT = TS_STATS * 16 * 8;
  static constexpr int BARS = (2 * TS_STAGES + 2 * 2 + 2 + 4 * TS_STATS + 1) * 8 + 8 + 4 * TS_STATS;
  static constexpr int BYTES = 128 + RING + COLS + STAT + BARS + TS_TILES;
};

// K-major operand without swizzle: 8-row x 16-byte core matrices, the ones along
// the rows 128 bytes apart, the ones along K TS_LBO.
__device__ __forceinline__ uint64_t ts_desc(uint32_t saddr) {
  return (uint64_t)((saddr & 0x3FFFFu) >> 4) | ((uint64_t)(TS_LBO >> 4) << 16) | ((uint64_t)(128 >> 4) << 32) |
         ((uint64_t)1 << 46);
}
// kind::f16, BF16 K-major operands, FP32 accumulate, 128 x n.
__device__ __forceinline__ uint32_t ts_idesc(int n) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(TS_BM >> 4) << 24);
}

// The next 8 significant bits of two values (lo half: x), and what is left of them.
__device__ __forceinline__ uint32_t ts_split(float& x, float& y) {
  uint32_t w;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(w) : "f"(y), "f"(x));
  x -= __uint_as_float(w << 16);
  y -= __uint_as_float(w & 0xffff0000u);
  return w;
}

__device__ __forceinline__ void ts_tmem_ld(uint32_t taddr, uint32_t (&r)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr));
}
__device__ __forceinline__ void ts_tmem_st(uint32_t taddr, const uint32_t (&r)[8]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"r"(taddr), "r"(r[0]),
               "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
               : "memory");
}

struct TsTile {
  int h, m0, n0;  // m0 in rows of A'
};
template <bool CPLX>
__device__ __forceinline__ TsTile ts_tile(const GemmArgs& g, int t, int tm, int tn) {
  constexpr int EM = CPLX ? TS_BM / 2 : TS_BM;
  const uint32_t r = (uint32_t)t / (uint32_t)tn, nt = (uint32_t)t - r * (uint32_t)tn;
  const uint32_t h = r / (uint32_t)tm, mt = r - h * (uint32_t)tm;
  return {(int)h, (int)mt * EM, (int)nt * TS_BN};
}

template <int BYTES>
__device__ __forceinline__ void ts_copy(uint32_t dst, const char* src, bool ok) {
  if constexpr (BYTES == 16)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(ok ? 16 : 0) : "memory");
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;" ::"r"(dst), "l"(src), "n"(BYTES), "r"(ok ? BYTES : 0)
                 : "memory");
}
// Producer of 32 plane rows of one operand: R operand rows x KQ depths per lane
// (lane / 4 along the rows, lane % 4 along the depth), so a lane's 8 plane depths
// of a row are one 16-byte store per plane.
template <bool CPLX, bool IS_A>
struct TsProducer {
  static constexpr int E = CPLX ? 2 : 1, ES = 4 * E, KQ = 8 / E, EK = TS_BK / E;
  static constexpr int R = CPLX && IS_A ? 2 : 4;
  static constexpr int V = 16 / ES;  // elements of a 16-byte load
  const GemmArgs& g;
  const int lane, c, row0;
  const bool by_rows;
  int ro[R];  // element offsets of the lane's rows (offsets fit 32 bits, launch_tc_stream)
  const char* base;
  bool rows_full;
  int koff;  // lane's: offset of depth k0 + lane of the next block to load

  __device__ __forceinline__ int64_t ld() const { return IS_A ? g.a_ld : g.b_ld; }
  __device__ __forceinline__ TsProducer(const GemmArgs& g_, int warp, int lane_)
      : g(g_), lane(lane_), c(lane_ & 3), row0((warp & 3) * 8 * R + (lane_ >> 2) * R),
        by_rows(IS_A ? g_.a_vec && !g_.a_kfast : g_.b_vec && !g_.b_kfast) {}

  __device__ __forceinline__ void tile(const TsTile& t) {
    const int nrows = (int)(IS_A ? g.M : g.N);
    const int64_t* rows = IS_A ? g.s.a_m : g.s.b_n;
    const int r0 = (IS_A ? t.m0 : t.n0) + row0;
#pragma unroll
    for (int i = 0; i < R; ++i) {
      const int r = min(r0 + i, nrows - 1);
      ro[i] = ld() ? r : __ldg(reinterpret_cast<const int*>(rows + r));
    }
    rows_full = __all_sync(0xffffffffu, r0 + R <= nrows);
    base = static_cast<const char*>(IS_A ? g.A : g.B) +
           (ld() ? (int64_t)t.h * g.K * ld() : __ldg((IS_A ? g.s.h_a : g.s.h_b) + t.h)) * ES;
  }
  __device__ __forceinline__ void fetch_k(int k0) {
    const int k = min(k0 + (lane < EK ? lane : 0), (int)g.K - 1);
    koff = ld() ? k * (int)ld() : __ldg(reinterpret_cast<const int*>((IS_A ? g.s.a_k : g.s.b_k) + k));
  }
  // The lane's elements of the block at k0 (koff fetched, the last depth's past K),
  // zero past K.
  __device__ __forceinline__ void load(float (&v)[R][8], int k0) const {
    const int kv = min(EK, (int)g.K - k0);
    const int kq = c * KQ;
    if (by_rows && rows_full) {
#pragma unroll
      for (int q = 0; q < KQ; ++q) {
        const int o = __shfl_sync(0xffffffffu, koff, kq + q);
#pragma unroll
        for (int i = 0; i < R; i += V) {
          float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
          if (kq + q < kv) x = __ldg(reinterpret_cast<const float4*>(base + (int64_t)(o + ro[i]) * ES));
          if constexpr (CPLX) {
            v[i][2 * q] = x.x;
            v[i][2 * q + 1] = x.y;
            v[i + 1][2 * q] = x.z;
            v[i + 1][2 * q + 1] = x.w;
          } else {
            v[i][q] = x.x;
            v[i + 1][q] = x.y;
            v[i + 2][q] = x.z;
            v[i + 3][q] = x.w;
          }
        }
      }
    } else if (!by_rows && (IS_A ? g.a_vec : g.b_vec) && kv == EK) {
      // by_rows is off, so the 16-byte groups run along the depth.
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const int o = __shfl_sync(0xffffffffu, koff, kq + j * V);
#pragma unroll
        for (int i = 0; i < R; ++i) {
          const float4 x = __ldg(reinterpret_cast<const float4*>(base + (int64_t)(o + ro[i]) * ES));
          v[i][4 * j] = x.x;
          v[i][4 * j + 1] = x.y;
          v[i][4 * j + 2] = x.z;
          v[i][4 * j + 3] = x.w;
        }
      }
    } else {
#pragma unroll
      for (int q = 0; q < KQ; ++q) {
        const int o = __shfl_sync(0xffffffffu, koff, kq + q);
#pragma unroll
        for (int i = 0; i < R; ++i) {
          const char* p = base + (int64_t)(o + ro[i]) * ES;
          if constexpr (CPLX) {
            float2 x = make_float2(0.f, 0.f);
            if (kq + q < kv) x = __ldg(reinterpret_cast<const float2*>(p));
            v[i][2 * q] = x.x;
            v[i][2 * q + 1] = x.y;
          } else {
            v[i][q] = kq + q < kv ? __ldg(reinterpret_cast<const float*>(p)) : 0.f;
          }
        }
      }
    }
  }

  // Splits one row's eight values into the planes. mx: the largest leading halves; mn:
  // the smallest non-zero magnitude as f32 bits, twice and less one (zero: the
  // largest). From the f32 bits: values of 2^-134 and below are zero in every plane.
  __device__ __forceinline__ void row(const float (&v)[8], char* d, uint32_t flip, uint32_t& mx, uint32_t& mn) const {
    uint32_t w[3][4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      float x = v[2 * j], y = v[2 * j + 1];
      mn = min(mn, min(2 * __float_as_uint(x) - 1, 2 * __float_as_uint(y) - 1));
      w[0][j] = ts_split(x, y);
      w[1][j] = ts_split(x, y);
      w[2][j] = ts_split(x, y);
      const uint32_t a = w[0][j] & 0x7fff7fffu;
      asm("max.u16x2 %0, %0, %1;" : "+r"(mx) : "r"(a));
    }
#pragma unroll
    for (int p = 0; p < 3; ++p) {
      if constexpr (CPLX && IS_A) {
        // Rows 2r: (re, -im); 2r + 1: (im, re).
        uint32_t e[4], o[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const uint32_t x = w[p][j] ^ flip;
          e[j] = x ^ 0x80000000u;
          o[j] = __byte_perm(x, x, 0x1032);
        }
        *reinterpret_cast<uint4*>(d + p * TS_PLANE) = make_uint4(e[0], e[1], e[2], e[3]);
        *reinterpret_cast<uint4*>(d + p * TS_PLANE + 16) = make_uint4(o[0], o[1], o[2], o[3]);
      } else {
        *reinterpret_cast<uint4*>(d + p * TS_PLANE) = make_uint4(w[p][0] ^ flip, w[p][1] ^ flip, w[p][2] ^ flip, w[p][3] ^ flip);
      }
    }
  }
  // Splits the lane's values into the operand's planes of a stage.
  __device__ __forceinline__ void split(const float (&v)[R][8], char* planes, uint32_t& mx, uint32_t& mn) const {
    constexpr int PR = CPLX && IS_A ? 2 : 1;  // plane rows per operand row
    // Core matrices of consecutive rows follow one another.
    char* d = planes + c * TS_LBO + PR * row0 * 16;
    const uint32_t flip = CPLX && (IS_A ? g.conj_a : g.conj_b) ? 0x80000000u : 0u;
#pragma unroll
    for (int i = 0; i < R; ++i) row(v[i], d + PR * i * 16, flip, mx, mn);
  }
};

template <bool CPLX, bool IS_A>
__device__ __forceinline__ void ts_produce(const GemmArgs& g, char* ring, uint64_t* full, uint64_t* empty, int2* stats,
                                           uint64_t* stat_full, uint64_t* stat_empty, int tiles, int tm, int tn,
                                           int warp, int lane) {
  using P = TsProducer<CPLX, IS_A>;
  P p(g, warp, lane);
  const int nk = (int)((g.K + P::EK - 1) / P::EK);
  // Whether this warp's rows of the tile exist (columns of B' past the product's width are not multiplied).
  const int first = (warp & 3) * 8 * P::R;
  uint32_t block = (uint32_t)warp >> 3;  // the set's blocks: every other one of the CTA's sequence
  int t = blockIdx.x, reported = t;  // the block's tile; the first tile whose range is not reported
  int kb = 0, it = 0;
  uint32_t mx = 0, mn = 0xffffffffu;
  bool act = false, ok = true;
  const auto advance = [&](int n) {
    kb += n;
    while (kb >= nk) {
      kb -= nk;
      t += gridDim.x;
    }
  };
  float v[P::R][8];
  const auto load = [&](bool new_tile) {
    if (t >= tiles) return;
    if (new_tile) {
      const TsTile x = ts_tile<CPLX>(g, t, tm, tn);
      p.tile(x);
      act = IS_A || x.n0 + first < g.N;
    }
    if (act) p.load(v, kb * P::EK);
    // The depth offsets of the set's block after this one.
    int k = kb + 2;
    while (k >= nk) k -= nk;
    p.fetch_k(k * P::EK);
  };
  // The value ranges of the tiles before `end`.
  const auto report = [&](int end) {
    for (; ok && reported < end; reported += gridDim.x, ++it) {
      const int s = it % TS_STATS;
      ok = __all_sync(0xffffffffu, mbar_wait_polls(&stat_empty[s], ((uint32_t)(it / TS_STATS) & 1u) ^ 1u));
      const int hi = (int)__reduce_max_sync(0xffffffffu, max(mx & 0xffffu, mx >> 16));
      const uint32_t lo = __reduce_min_sync(0xffffffffu, mn);
      if (lane == 0 && ok) {
        stats[s * 16 + warp] = make_int2(hi, lo == 0xffffffffu ? 0x7fff : (int)((lo + 1) >> 17));
        mbar_arrive(&stat_full[s]);
      }
      __syncwarp();
      mx = 0;
      mn = 0xffffffffu;
    }
  };
  advance((int)block);
  p.fetch_k(kb * P::EK);
  load(true);
  while (t < tiles) {
    report(t);
    const uint32_t stage = block % TS_STAGES, round = block / TS_STAGES;
    ok = ok && mbar_wait_polls(&empty[stage], (round & 1u) ^ 1u);
    ok = __all_sync(0xffffffffu, ok);
    if (!ok) break;
    if (act) p.split(v, ring + stage * TS_STAGE + (IS_A ? 0 : 3 * TS_PLANE), mx, mn);
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncwarp();
    if (lane == 0) mbar_arrive(&full[stage]);
    // The next block's elements are on their way while the other set splits.
    const int told = t;
    advance(2);
    load(t != told);
    block += 2;
  }
  report(tiles);
  if (!ok) atomicOr(g.status, STATUS_WAIT_TIMEOUT);
}

__device__ __forceinline__ void ts_mark(unsigned char* again, int tile, int warp) {
  atomicOr(reinterpret_cast<uint32_t*>(again + (tile & ~3)), 1u << (8 * (tile & 3) + warp));
}

// STEPS: steps of 16 plane depths (one MMA each) in all of K: 1, 2 or (3) more.
// GEN: D is more than the sums (alpha, C, conjugation), an instantiation of its own, as
// the registers for C cost the other calls a tenth.
template <bool CPLX, int STEPS, bool GEN>
__global__ void __launch_bounds__(TS_THREADS, 1) tc_stream_kernel(const __grid_constant__ GemmArgs g, int tiles, int tm,
                                                                  int tn, unsigned char* __restrict__ flags) {
  constexpr int E = CPLX ? 2 : 1, EK = TS_BK / E;
  extern __shared__ unsigned char ts_smem[];
  char* ring = reinterpret_cast<char*>((reinterpret_cast<uintptr_t>(ts_smem) + 127) & ~uintptr_t(127));
  int64_t* cols = reinterpret_cast<int64_t*>(ring + TsSmem::RING);
  int2* stats = reinterpret_cast<int2*>(ring + TsSmem::RING + TsSmem::COLS);
  uint64_t* full = reinterpret_cast<uint64_t*>(ring + TsSmem::RING + TsSmem::COLS + TsSmem::STAT);
  uint64_t* empty = full + TS_STAGES;
  uint64_t* main_full = empty + TS_STAGES;
  uint64_t* main_empty = main_full + 2;
  uint64_t* corr_empty = main_empty + 2;
  uint64_t* stat_full = corr_empty + 2;
  uint64_t* stat_empty = stat_full + TS_STATS;
  uint64_t* thr_full = stat_empty + TS_STATS;
  uint64_t* thr_empty = thr_full + TS_STATS;
  uint64_t* done = thr_empty + TS_STATS;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(done + 1);
  // Per tile of this CTA, the epilogue warps whose outputs are computed again.
  volatile float* thresholds = reinterpret_cast<float*>(tmem_slot + 2);  // split_guard of a tile
  unsigned char* again = reinterpret_cast<unsigned char*>(tmem_slot + 2 + TS_STATS);
  const int mine = (tiles - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x;

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int nk = (int)((g.K + EK - 1) / EK);
  if (tid == 0) {
    for (int s = 0; s < TS_STAGES; ++s) {
      mbar_init(&full[s], 8);
      mbar_init(&empty[s], 1);
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(&main_full[s], 1);
      mbar_init(&main_empty[s], 8);
      mbar_init(&corr_empty[s], 8);
    }
    for (int s = 0; s < TS_STATS; ++s) {
      mbar_init(&stat_full[s], 16);
      mbar_init(&stat_empty[s], 1);
      mbar_init(&thr_full[s], 1);
      mbar_init(&thr_empty[s], 8);
    }
    mbar_init(done, 1);
    fence_barrier_init();
  }
  if (warp == 24) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  for (int i = 4 * threadIdx.x; i < mine; i += 4 * TS_THREADS) *reinterpret_cast<uint32_t*>(again + i) = 0;
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  // Tensor memory, 128 columns each, per STEPS. 1: two sets of the leading products and
  // the cross products. 2: the leading products of either step, and the cross products
  // of two tiles. 3: those of a block's steps, the cross products, the running sum.
  constexpr bool MULTI = STEPS == 3;
  const int steps_all = (int)((g.K * (CPLX ? 2 : 1) + 15) / 16);
  const uint32_t tmem = *tmem_slot;

  // Registers a thread: 64 x 256 + 80 x 512 + 56 x 128 = 64512, the launch's 72 x 896.
  if (warp >= 8 && warp < 24) {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 80;");
    if ((warp & 7) < 4)
      ts_produce<CPLX, true>(g, ring, full, empty, stats, stat_full, stat_empty, tiles, tm, tn, warp - 8, lane);
    else
      ts_produce<CPLX, false>(g, ring, full, empty, stats, stat_full, stat_empty, tiles, tm, tn, warp - 8, lane);
  } else if (warp >= 24) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 56;");
    if (warp == 24 && lane == 0) {
      int stage = 0;
      uint32_t round = 0, blocks = 0;
      bool ok = true;
      int it = 0;
      for (int t = blockIdx.x; ok && t < tiles; t += gridDim.x, ++it) {
        const TsTile x = ts_tile<CPLX>(g, t, tm, tn);
        const int n = min(TS_BN, ((int)g.N - x.n0 + 15) / 16 * 16);
        const uint32_t idesc = ts_idesc(n);
        const int set = MULTI ? 0 : it & 1, mset = STEPS == 1 ? set : 0;
        const uint32_t main0 = tmem + 256 * mset, main1 = main0 + 128,
                       corr = STEPS == 1 ? main1 : tmem + 256 + 128 * set;
        const uint32_t tile_turn = (uint32_t)(MULTI ? it : it >> 1);
        if (!mbar_wait_polls(&corr_empty[set], (tile_turn & 1u) ^ 1u)) ok = false;
        for (int kb = 0; ok && kb < nk; ++kb, ++blocks) {
          if (!mbar_wait_polls(&full[stage], round & 1u)) {
            ok = false;
            break;
          }
          tc_fence_after();
          const uint32_t sa = smem_u32(ring + stage * TS_STAGE), sb = sa + 3 * TS_PLANE;
          const int steps = min(2, steps_all - 2 * kb);
          for (int kk = 0; kk < steps; ++kk) {
            uint64_t a[3], b[3];
#pragma unroll
            for (int p = 0; p < 3; ++p) {
              a[p] = ts_desc(sa + p * TS_PLANE + 2 * kk * TS_LBO);
              b[p] = ts_desc(sb + p * TS_PLANE + 2 * kk * TS_LBO);
            }
            umma_bf16(corr, a[1], b[2], idesc, (kb | kk) != 0 ? 1u : 0u);
            umma_bf16(corr, a[2], b[1], idesc, 1u);
            umma_bf16(corr, a[0], b[2], idesc, 1u);
            umma_bf16(corr, a[2], b[0], idesc, 1u);
            umma_bf16(corr, a[1], b[1], idesc, 1u);
            umma_bf16(corr, a[0], b[1], idesc, 1u);
            umma_bf16(corr, a[1], b[0], idesc, 1u);
          }
          // The leading products of the block before have been read.
          if (!mbar_wait_polls(&main_empty[mset], ((STEPS == 1 ? tile_turn : blocks) & 1u) ^ 1u)) {
            ok = false;
            break;
          }
          tc_fence_after();
          umma_bf16(main0, ts_desc(sa), ts_desc(sb), idesc, 0u);
          if (steps == 2) umma_bf16(main1, ts_desc(sa + 2 * TS_LBO), ts_desc(sb + 2 * TS_LBO), idesc, 0u);
          umma_commit(&empty[stage]);
          umma_commit(&main_full[mset]);
          if (++stage == TS_STAGES) {
            stage = 0;
            ++round;
          }
        }
      }
      if (!ok) atomicOr(g.status, STATUS_WAIT_TIMEOUT);
      // Nothing of this CTA's tensor work is in flight when it ends.
      umma_commit(done);
      if (!mbar_wait_polls(done, 0)) atomicOr(g.status, STATUS_WAIT_TIMEOUT);
    }
    __syncwarp();
    if (warp == 25) {
      // The tiles' thresholds from the value ranges that the producers found.
      bool ok = true;
      for (int it = 0; ok && it < mine; ++it) {
        const int s = it % TS_STATS;
        const uint32_t turn = (uint32_t)(it / TS_STATS);
        ok = mbar_wait_polls(&stat_full[s], turn & 1u) && mbar_wait_polls(&thr_empty[s], (turn & 1u) ^ 1u);
        ok = __all_sync(0xffffffffu, ok);
        const int2 r = stats[s * 16 + (lane & 15)];
        const bool is_a = (lane & 4) == 0;
        const int amax = (int)__reduce_max_sync(0xffffffffu, (uint32_t)(is_a ? r.x : 0));
        const int bmax = (int)__reduce_max_sync(0xffffffffu, (uint32_t)(is_a ? 0 : r.x));
        const int amin = (int)__reduce_min_sync(0xffffffffu, (uint32_t)(is_a ? r.y : 0x7fff));
        const int bmin = (int)__reduce_min_sync(0xffffffffu, (uint32_t)(is_a ? 0x7fff : r.y));
        if (lane == 0 && ok) {
          thresholds[s] = split_guard((amax >> 7) - 127, amin == 0x7fff ? 999 : (amin >> 7) - 127, (bmax >> 7) - 127,
                                      bmin == 0x7fff ? 999 : (bmin >> 7) - 127, (int)g.K * (CPLX ? 2 : 1));
          mbar_arrive(&stat_empty[s]);
          mbar_arrive(&thr_full[s]);
        }
        __syncwarp();
      }
      if (!ok) atomicOr(g.status, STATUS_WAIT_TIMEOUT);
      __syncwarp();
    }
  } else {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 64;");
    const int col0 = (warp >> 2) * TS_CPT;
    int64_t* cols_w = cols + warp * 4 * TS_CPT;
    const uint32_t lane_addr = ((uint32_t)(32 * (warp & 3)) << 16) + col0;
    const int prow = 32 * (warp & 3) + lane, comp = CPLX ? prow & 1 : 0;
    const Epilogue e = g.e;
    uint32_t blocks = 0;
    int it = 0;
    bool ok = true;
    float sums[MULTI ? TS_CPT : 1];  // of TS_FLUSH blocks each
    // Output offsets of a tile, fetched while the one before it is written back.
    int64_t nd = 0, nc = 0;
    const auto fetch = [&](const TsTile& x, int buf) {
      const int m = min(x.m0 + (CPLX ? prow >> 1 : prow), (int)g.M - 1);
      nd = __ldg(g.s.d_m + m) + __ldg(g.s.h_d + x.h);
      if (!e.beta_zero) nc = __ldg(g.s.c_m + m) + __ldg(g.s.h_c + x.h);
#pragma unroll
      for (int j = 0; j < TS_CPT / 32; ++j) {
        const int n = min(x.n0 + col0 + lane + 32 * j, (int)g.N - 1);
        const uint32_t d = smem_u32(cols_w + buf * 2 * TS_CPT + lane + 32 * j);
        ts_copy<8>(d, reinterpret_cast<const char*>(g.s.d_n + n), true);
        if (!e.beta_zero) ts_copy<8>(d + TS_CPT * 8, reinterpret_cast<const char*>(g.s.c_n + n), true);
      }
    };
    fetch(ts_tile<CPLX>(g, blockIdx.x, tm, tn), 0);
    for (int t = blockIdx.x; ok && t < tiles; t += gridDim.x, ++it) {
      const TsTile x = ts_tile<CPLX>(g, t, tm, tn);
      const int m = x.m0 + (CPLX ? prow >> 1 : prow), n0 = x.n0 + col0;
      const bool mok = m < (int)g.M;
      const int nrem = max(0, min(TS_CPT, (int)g.N - n0));
      // A lane writes one component of its row.
      float* const Db = static_cast<float*>(g.D) + nd * E + comp;
      const float* const Cb = static_cast<const float*>(g.C) + nc * E + comp;
      const int64_t *dn_s = cols_w + (it & 1) * 2 * TS_CPT, *cn_s = dn_s + TS_CPT;
      asm volatile("cp.async.wait_all;" ::: "memory");
      __syncwarp();
      if (t + (int)gridDim.x < tiles) fetch(ts_tile<CPLX>(g, t + gridDim.x, tm, tn), (it + 1) & 1);
      const int set = MULTI ? 0 : it & 1, mset = STEPS == 1 ? set : 0;
      const uint32_t main0 = tmem + 256 * mset + lane_addr, main1 = main0 + 128,
                     corr = STEPS == 1 ? main1 : tmem + 256 + 128 * set + lane_addr, total = tmem + 384 + lane_addr;
      // All blocks but the last into the running sum, which starts again every
      // TS_FLUSH blocks, so that the roundings of a long K do not pile up.
      for (int kb = 0; MULTI && kb + 1 < nk; ++kb, ++blocks) {
        if (!mbar_wait_polls(&main_full[0], blocks & 1u)) {
          ok = false;
          break;
        }
        tc_fence_after();
        const bool first = kb % TS_FLUSH == 0, last = kb % TS_FLUSH == TS_FLUSH - 1;
#pragma unroll 1
        for (int q = 0; 8 * q < nrem; ++q) {
          uint32_t r[8], u[8], w[8];
          ts_tmem_ld(main0 + 8 * q, r);
          ts_tmem_ld(main1 + 8 * q, u);
          ts_tmem_ld(total + 8 * q, w);
          tmem_ld_wait(r, u, w);
#pragma unroll
          for (int j = 0; j < 8; ++j)
            r[j] = __float_as_uint((first ? 0.f : __uint_as_float(w[j])) + (__uint_as_float(r[j]) + __uint_as_float(u[j])));
          if (last) {
#pragma unroll
            for (int j = 0; j < 8; ++j)
              sums[8 * q + j] = (kb == TS_FLUSH - 1 ? 0.f : sums[8 * q + j]) + __uint_as_float(r[j]);
          } else {
            ts_tmem_st(total + 8 * q, r);
          }
        }
        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&main_empty[0]);
      }
      // The last block, whose commit covers the cross products; then the value ranges
      // of the tile's operands.
      const int s = it % TS_STATS;
      if (ok) ok = mbar_wait_polls(&main_full[mset], (STEPS == 1 ? (uint32_t)(it >> 1) : blocks) & 1u);
      if (ok) ok = mbar_wait_polls(&thr_full[s], (uint32_t)(it / TS_STATS) & 1u);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      tc_fence_after();
      const float thr = thresholds[s];
      const bool second = steps_all % 2 == 0, more = (nk - 1) % TS_FLUSH != 0, flushed = nk > TS_FLUSH;
      // Sums that the planes may not carry are computed again: all of them, or (a finite
      // threshold, and D only written) this warp's once one of them is below it.
      const bool skip = thr == __uint_as_float(0x7f800000u) || (thr != 0.f && GEN);
      if (skip && lane == 0) ts_mark(again, it, warp);
      const int ncols = skip ? 0 : nrem;
      float least = __uint_as_float(0x7f800000u);  // magnitude of what this lane writes
      // C of eight columns, a group ahead of its use.
      float cv[GEN ? 8 : 1], cnext[GEN ? 8 : 1];
      const auto fetch_c = [&](int q) {
        if constexpr (GEN) {
          if (e.beta_zero) return;
#pragma unroll
          for (int j = 0; j < 8; ++j) cnext[j] = mok && 8 * q + j < ncols ? Cb[cn_s[8 * q + j] * E] : 0.f;
        }
      };
      if constexpr (GEN) {
#pragma unroll
        for (int j = 0; j < 8; ++j) cnext[j] = 0.f;
        fetch_c(0);
      }
#pragma unroll 1
      for (int q = 0; 8 * q < ncols; ++q) {
        {
          uint32_t r[8], u[8];
          float v[8];
          if constexpr (GEN) {
#pragma unroll
            for (int j = 0; j < 8; ++j) cv[j] = cnext[j];
            fetch_c(q + 1);
          }
          ts_tmem_ld(main0 + 8 * q, r);
          ts_tmem_ld(main1 + 8 * q, u);  // STEPS 1: the cross products
          if constexpr (MULTI) {
            uint32_t w[8];
            ts_tmem_ld(total + 8 * q, w);
            tmem_ld_wait(r, u, w);
#pragma unroll
            for (int j = 0; j < 8; ++j)
              v[j] = __uint_as_float(r[j]) + (second ? __uint_as_float(u[j]) : 0.f) + (more ? __uint_as_float(w[j]) : 0.f);
            ts_tmem_ld(corr + 8 * q, u);
            if (flushed) {
#pragma unroll
              for (int j = 0; j < 8; ++j) v[j] += sums[8 * q + j];
            }
            tmem_ld_wait(u);
          } else if constexpr (STEPS == 2) {
            uint32_t w[8];
            ts_tmem_ld(corr + 8 * q, w);
            tmem_ld_wait(r, u, w);
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              v[j] = __uint_as_float(r[j]) + __uint_as_float(u[j]);
              u[j] = w[j];
            }
          } else {
            tmem_ld_wait(r, u);
#pragma unroll
            for (int j = 0; j < 8; ++j) v[j] = __uint_as_float(r[j]);
          }
#pragma unroll
          for (int j = 0; j < 8; ++j) v[j] += __uint_as_float(u[j]);
          if constexpr (GEN) {
            // D = op(alpha acc + beta op(C)) of this lane's component; the other one of a
            // complex row sits in the neighbouring lane.
            const float ar = (float)e.alpha_re, ai = comp ? (float)e.alpha_im : -(float)e.alpha_im;
            const float br = (float)e.beta_re, bi = comp ? (float)e.beta_im : -(float)e.beta_im;
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              float y = v[j] * ar;
              if constexpr (CPLX) y += __shfl_xor_sync(0xffffffffu, v[j], 1) * ai;
              if (!e.beta_zero) {
                const float c = CPLX && e.conj_c && comp ? -cv[j] : cv[j];
                y += c * br;
                if constexpr (CPLX) y += __shfl_xor_sync(0xffffffffu, c, 1) * bi;
              }
              v[j] = CPLX && e.conj_d && comp ? -y : y;
            }
          } else {
#pragma unroll
            for (int j = 0; j < 8; ++j)
              if (8 * q + j < ncols) least = fminf(least, fabsf(v[j]));
          }
          if (mok) {
            if (8 * q + 8 <= ncols) {
#pragma unroll
              for (int j = 0; j < 8; j += 2) {
                const longlong2 o = *reinterpret_cast<const longlong2*>(dn_s + 8 * q + j);
                Db[o.x * E] = v[j];
                Db[o.y * E] = v[j + 1];
              }
            } else {
#pragma unroll
              for (int j = 0; j < 8; ++j)
                if (8 * q + j < ncols) Db[dn_s[8 * q + j] * E] = v[j];
            }
          }
          __syncwarp();
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) {
        mbar_arrive(&main_empty[mset]);
        mbar_arrive(&corr_empty[set]);
      }
      const float bound = thresholds[s];
      if (bound != 0.f && !skip && __any_sync(0xffffffffu, !(least >= bound)) && lane == 0) ts_mark(again, it, warp);
      __syncwarp();
      if (lane == 0) mbar_arrive(&thr_empty[s]);
      ++blocks;
    }
    if (!ok) atomicOr(g.status, STATUS_WAIT_TIMEOUT);
    __syncwarp();
  }

  tc_fence_before();
  __syncthreads();
  for (int i = tid; i < mine; i += TS_THREADS) flags[blockIdx.x + i * gridDim.x] = again[i];
  if (warp == 24) {
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
}

// Copy of an operand into a dense panel [H][K][ld], rows fastest: 32 rows by 32 of
// the index that is fastest in memory (depth or batch; FAST 0: rows, with 32
// depths) per CTA, through shared memory.
template <class T, int FAST>
__global__ void __launch_bounds__(256) stream_pack_kernel(const T* __restrict__ X, const int64_t* __restrict__ rows,
                                                          const int64_t* __restrict__ ks, const int64_t* __restrict__ hs,
                                                          int64_t nrows, int64_t K, int64_t H, int64_t ld,
                                                          T* __restrict__ out) {
  __shared__ T tile[32][33];
  // The second index of a tile: the batch (FAST 2) or the depth; `o` the other.
  const int64_t n2 = FAST == 2 ? H : K, no = FAST == 2 ? K : H;
  const int64_t* s2 = FAST == 2 ? hs : ks;
  const int64_t* so = FAST == 2 ? ks : hs;
  const int64_t tr = (nrows + 31) / 32, t2 = (n2 + 31) / 32;
  const int x = threadIdx.x & 31, y = threadIdx.x >> 5;
  for (int64_t t = blockIdx.x; t < tr * t2 * no; t += gridDim.x) {
    const int64_t r0 = t % tr * 32, q0 = t / tr % t2 * 32, o = t / tr / t2;
    const T* base = X + so[o];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int rr = FAST ? y + 8 * j : x, q = FAST ? x : y + 8 * j;
      if (r0 + rr < nrows && q0 + q < n2) tile[q][rr] = base[rows[r0 + rr] + s2[q0 + q]];
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int q = y + 8 * j;
      if (r0 + x < nrows && q0 + q < n2)
        out[(FAST == 2 ? (q0 + q) * K + o : o * K + q0 + q) * ld + r0 + x] = tile[q][x];
    }
    __syncthreads();
  }
}
int64_t panel_ld(int64_t rows) { return (rows + 15) / 16 * 16; }

template <class T>
void run_stream_pack(const GemmArgs& g, int which, int fast, int64_t ld, void* panel, cudaStream_t st) {
  const bool a = which == 0;
  const int64_t rows = a ? g.M : g.N;
  const int64_t tiles = ((rows + 31) / 32) * (fast == 2 ? (g.H + 31) / 32 * g.K : (g.K + 31) / 32 * g.H);
  const unsigned grid = (unsigned)(tiles < 8192 ? tiles : 8192);
  auto kern = fast == 2 ? stream_pack_kernel<T, 2> : fast == 1 ? stream_pack_kernel<T, 1> : stream_pack_kernel<T, 0>;
  kern<<<grid, 256, 0, st>>>(static_cast<const T*>(a ? g.A : g.B), a ? g.s.a_m : g.s.b_n, a ? g.s.a_k : g.s.b_k,
                             a ? g.s.h_a : g.s.h_b, rows, g.K, g.H, ld, static_cast<T*>(panel));
}

}  // namespace

bool is_tc_stream(int kernel) { return kernel == PLAIN_F32_TC_STREAM || kernel == PLAIN_C32_TC_STREAM; }

size_t stream_panel_bytes(int dtype, int64_t rows, int64_t K, int64_t H) {
  return (size_t)H * K * panel_ld(rows) * (dtype == 0 ? 4 : 8) + 256;
}

cudaError_t launch_stream_pack(int dtype, GemmArgs& g, int which, int fast, void* panel, cudaStream_t st) {
  const bool a = which == 0;
  const int64_t ld = panel_ld(a ? g.M : g.N);
  if (dtype == 0)
    run_stream_pack<float>(g, which, fast, ld, panel, st);
  else if (dtype == 2)
    run_stream_pack<float2>(g, which, fast, ld, panel, st);
  else
    return cudaErrorInvalidValue;
  if (a) {
    g.A = panel;
    g.a_ld = ld;
    g.a_kfast = 0;
    g.a_vec = 1;
  } else {
    g.B = panel;
    g.b_ld = ld;
    g.b_kfast = 0;
    g.b_vec = 1;
  }
  return cudaGetLastError();
}

// Index arithmetic of the kernel: rows, depths and tiles in 32 bits, and an
// operand's row plus depth offset (in its panel, where it is packed) as well.
bool tc_stream_fits(int dtype, int64_t M, int64_t N, int64_t K, int64_t H, const LaunchHints& hints) {
  constexpr int64_t most = (int64_t)1 << 30;
  if (dtype != 0 && dtype != 2) return false;
  if (!hints.known || !hints.off32 || K <= 0 || K >= most || M >= most || N >= most || H >= most) return false;
  if ((!hints.a_gather && (double)panel_ld(M) * (double)K >= 2.0 * most - (double)M) ||
      (!hints.b_gather && (double)panel_ld(N) * (double)K >= 2.0 * most - (double)N))
    return false;
  const int64_t em = dtype == 2 ? TS_BM / 2 : TS_BM;
  const double tiles = (double)TS_TILES * 64;  // TS_TILES for each CTA of a grid of 64 or more
  return ((double)(M / em) + 1) * ((double)(N / TS_BN) + 1) * (double)H < tiles &&
         ((double)(N / em) + 1) * ((double)(M / TS_BN) + 1) * (double)H < tiles;
}

// Against the FFMA families by estimated microseconds. Fitted on B200 to 600 contractions
// (matrix products, batches, permuted, six-index and transformation shapes, K from 1 to
// 4096) timed on all three; typical deviation 7 to 12 %. The family chosen is 4.3 % above
// the best of the three in the geometric mean (with constants fitted to an earlier state
// of the kernels 7.7 %). Below 2^23 products the launches decide.
//
// FFMA: the choice made without these families, by its tile waves, with the pack pass, the
// write-back and split K. In flight: waves of tiles, stages of 32 plane depths, panels.
// Packed: the planes' bytes, waves of 128 x 256 tiles by plane depth (a partial wave in
// parts). Each with a constant for its launches, and with the operand elements that a
// panel or the planes read uncoalesced.
//
// With tiles for less than a quarter of the SMs, near a tie, the FFMA families' one launch
// takes the call. From a quarter up these
// families keep what is estimated within 7 us of FFMA: their sums are the more accurate,
// and the estimate of a call this short is off by as much (f32 2564 x 129 x 128: estimated
// 7 apart, measured 14.4 to 16.5 FFMA, 18.5 here).
int choose_tc_kernel(int dtype, int64_t M, int64_t N, int64_t K, int64_t H, int num_sms, const LaunchHints& hints) {
  if (!hints.tensor || !tc_stream_fits(dtype, M, N, K, H, hints)) return 0;
  const bool cplx = dtype == 2;
  const int64_t m = hints.d_mfast ? M : N, n = hints.d_mfast ? N : M;  // the launch's roles
  const int64_t em = cplx ? TS_BM / 2 : TS_BM, ek = cplx ? TS_BK / 2 : TS_BK, e = cplx ? 2 : 1;
  const int64_t tiles = ((m + em - 1) / em) * ((n + TS_BN - 1) / TS_BN) * H;
  const double outs = (double)M * (double)N * (double)H, k = (double)K;
  if (tiles < 16 || outs * k * (cplx ? 4 : 1) < (double)(1 << 23)) return 0;

  LaunchHints general = hints;
  general.tensor = false;
  int kernel = 0, splits = 1, bm = 0, bn = 0;
  int64_t chunk = 0;
  choose_plain_launch(dtype, 0, M, N, K, H, num_sms, general, &kernel, &splits, &chunk);
  plain_tile_shape(kernel, &bm, &bn);
  const double rows = (double)((M + bm - 1) / bm * bm), cols = (double)((N + bn - 1) / bn * bn);
  const double area = (double)bm * bn, whole = rows / bm * (cols / bn) * (double)H * splits;
  double ffma;
  if (is_packed_kernel(kernel)) {
    const double slots = (cplx ? 2 : 1) * (double)num_sms, w = whole < 3 * slots ? std::ceil(whole / slots) : whole / slots + 0.5;
    const double bytes = 4 * (rows * (cplx ? 4 : 1) + cols * (cplx ? 2 : 1)) * k * (double)H, part = std::ceil(k / splits);
    ffma = cplx ? 10.2 + 0.53e-6 * bytes + w * 0.154 * part + (splits > 1 ? 11.2e-6 * splits * outs : 0) + 10.7e-6 * outs
                : 6.7 + 0.55e-6 * bytes + w * (0.074 * part + 8.3) + (splits > 1 ? 5.6 + 1.6e-6 * splits * outs : 0) + 3.6e-6 * outs;
  } else {
    const double w = std::max(1.0, whole / num_sms) * area * k * 1e-6, t = std::max(1.0, whole / num_sms);
    ffma = cplx ? 5.2 + 8.7 * 4 * w + 3.5 * t + 1.9e-6 * outs
           : bm == 128 ? 10.8 + 11.2 * w + 5.4 * t + 1.2e-6 * outs
                       : 5.2 + 15.0 * w + 1.3 * t + 3.3e-6 * outs;
    ffma = std::max(9.0, ffma);
  }

  const double waves = (double)((tiles + num_sms - 1) / num_sms), stages = (double)((K + ek - 1) / ek);
  const int panels = (hints.a_gather ? 0 : 1) + (hints.b_gather ? 0 : 1);
  const double panel = ((hints.a_gather ? 0 : (double)M) + (hints.b_gather ? 0 : (double)N)) * k * (double)H;
  const double width = std::min(1.0, std::max((double)n, 8.0) / TS_BN);
  const double here = cplx ? 8.5 + waves * (2.0 * width + 0.27 + 1.64 * stages) + 3.7 * panels + 6.2e-6 * panel + 0.44e-6 * outs
                           : 9.4 + waves * (1.5 * width + 0.23 + 2.0 * stages) + 3.4 * panels + 5.3e-6 * panel + 0.18e-6 * outs;

  double split = 1e30;
  if (tc_split_fits(dtype, M, N, K, H)) {
    const int64_t mp = (m * e + 127) / 128 * 128, np = (n + 255) / 256 * 256, kp = (K * e + 63) / 64 * 64;
    const int64_t t = mp / 128 * (np / 256) * H, rem = t % num_sms;
    double w;
    if (t >= num_sms)
      w = (double)(t / num_sms) + (rem ? 1.0 / (double)std::max<int64_t>(1, std::min<int64_t>(4, num_sms / rem)) : 0.0);
    else
      w = 1.0 / (double)std::max<int64_t>(1, std::min<int64_t>(std::min<int64_t>(16, num_sms / t), kp / 64));
    const double bytes = ((double)(mp + np) * (double)kp * 6 + (double)(m + n) * k * 4 * (double)e) * (double)H;
    split = cplx ? 19.8 + 0.405e-6 * bytes + 1.55e-6 * panel + 0.0322 * w * (double)kp + 6.8 * std::ceil(w) + 1.9e-6 * outs
                 : 15.2 + 0.38e-6 * bytes + 2.1e-6 * panel + 0.045 * w * (double)kp + 10.7 * std::ceil(w) + 0.27e-6 * outs;
  }
  const double bar = tiles * 4 < num_sms ? 0.95 * ffma : ffma + 7.0;
  if (std::min(here, split) >= bar) return 0;
  if (split < here) return cplx ? PLAIN_C32_TC_SPLIT : PLAIN_F32_TC_SPLIT;
  return cplx ? PLAIN_C32_TC_STREAM : PLAIN_F32_TC_STREAM;
}

// The caller has checked tc_stream_fits.
size_t tc_stream_flag_bytes(int dtype, int64_t M, int64_t N, int64_t H) {
  const auto tiles = [&](int64_t m, int64_t n) { return ((m + (dtype == 2 ? 63 : 127)) / (dtype == 2 ? 64 : 128)) * ((n + TS_BN - 1) / TS_BN) * H; };
  return (size_t)std::max(tiles(M, N), tiles(N, M)) + 256;  // either orientation
}

cudaError_t launch_tc_stream(int dtype, const GemmArgs& g, void* flags, cudaStream_t st) {
  if (dtype != 0 && dtype != 2) return cudaErrorInvalidValue;
  const int64_t em = dtype == 2 ? TS_BM / 2 : TS_BM;
  const int64_t tm = (g.M + em - 1) / em, tn = (g.N + TS_BN - 1) / TS_BN, tiles = tm * tn * g.H;
  int dev = 0, sms = 148;
  if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const unsigned grid = (unsigned)(tiles < sms ? tiles : sms);
  const int64_t steps = (g.K * (dtype == 2 ? 2 : 1) + 15) / 16;
  const auto pick = [&](auto cplx, auto gen) {
    constexpr bool C = decltype(cplx)::value, G = decltype(gen)::value;
    return steps == 1 ? tc_stream_kernel<C, 1, G> : steps == 2 ? tc_stream_kernel<C, 2, G> : tc_stream_kernel<C, 3, G>;
  };
  const auto of = [&](auto cplx) { return g.e.plain ? pick(cplx, std::false_type{}) : pick(cplx, std::true_type{}); };
  auto kern = dtype == 2 ? of(std::true_type{}) : of(std::false_type{});
  const cudaError_t r = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, TsSmem::BYTES);
  if (r != cudaSuccess) return r;
  kern<<<grid, TS_THREADS, TsSmem::BYTES, st>>>(g, (int)tiles, (int)tm, (int)tn, static_cast<unsigned char*>(flags));
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  return launch_ffma_again(dtype, g, static_cast<const unsigned char*>(flags), tiles, tm, tn, TS_BN, false, sms, st);
}

}  // namespace dev
}  // namespace tprims
