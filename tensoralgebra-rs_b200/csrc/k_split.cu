// Split-precision f32 contraction on the sm_100a tensor cores.
//
// f32 operands are split into BF16 planes, x = x0 + x1 (+ x2), and the
// product is accumulated in FP32 from a subset of the plane products:
//   bf16x3: x0*y0 + x0*y1 + x1*y0                       (2 planes, 3 products)
//   bf16x6: bf16x3 + x0*y2 + x1*y1 + x2*y0              (3 planes, 6 products)
// Each plane keeps the next 8 significant bits of the remainder, so bf16x6
// carries 24 bits (the f32 significand) and drops x1*y2 + x2*y1 and less, at
// most 2^-24 of the product; bf16x3 carries 16 bits.
//
// Two kernels:
//  * split_pack: gathers A' (or B') through its scatter vectors (the packing of
//    crates/tprims-kernel/src/pack/pack.rs:152-203, here into HBM once per
//    call), transposes through shared memory so that reads run along the
//    operand's unit-stride index and writes along k, splits, and writes the
//    planes K-major, zero-padded to whole tiles.
//  * tc_bf16_gemm: one CTA per 128 x BN output tile. Warp 0 issues TMA tile
//    loads (SWIZZLE_64B, 32 k per stage) into a multi-stage ring; warp 1 owns
//    the TMEM accumulators and issues tcgen05.mma kind::f16 (BF16 in, FP32
//    accumulate) from one thread; warps 2-9 drain the accumulators with
//    tcgen05.ld into FP32 registers (two-level accumulation, see below) and
//    apply the scatter epilogue D = op_D(alpha*acc + beta*C)
//    (pack/writeback.rs:311-486). Every mbarrier wait is bounded by
//    %globaltimer; a timeout sets a status bit and the kernel drains and
//    returns. No cluster, no multicast.
//
// The same GEMM serves plain f32 and c32 contractions that are large enough to pay
// for the planes' pass through HBM (PLAIN 1 and 2; smaller ones split on the way into
// shared memory, k_tcstream.cu). c32 is embedded as the real product of 2M x N x 2K.
// plain_split_pack_kernel also notes the range of the values it splits; outputs that
// the planes may not carry to f32 rounding (split_guard) are computed again by FFMA.
#include <cuda.h>
#include <cuda_bf16.h>

#include <type_traits>

#include "tc_common.cuh"

namespace tprims {
namespace dev {

namespace {

using namespace tc;

constexpr int TC_BM = 128;
constexpr int TC_BK = 32;  // BF16 elements per stage row: 64 bytes = one SWIZZLE_64B atom

// Instruction descriptor of kind::f16: BF16 A and B (K-major), FP32 D, M x N.
__host__ __device__ constexpr uint32_t idesc_bf16(int M, int N) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

__device__ inline void split3(float x, __nv_bfloat16& p0, __nv_bfloat16& p1, __nv_bfloat16& p2) {
  p0 = __float2bfloat16_rn(x);
  const float r1 = x - __bfloat162float(p0);
  p1 = __float2bfloat16_rn(r1);
  const float r2 = r1 - __bfloat162float(p1);
  p2 = __float2bfloat16_rn(r2);
}

// Gather + split + K-major write of one 32-row x 64-k tile.
__global__ void __launch_bounds__(256) split_pack_kernel(const float* __restrict__ X, const int64_t* __restrict__ rows_scat,
                                                         const int64_t* __restrict__ k_scat,
                                                         const int64_t* __restrict__ h_scat,
                                                         const int64_t* __restrict__ rows_blk,
                                                         const int64_t* __restrict__ k_blk, int64_t nrows, int64_t K,
                                                         int64_t rows_pad, int64_t k_pad, int64_t H, int kfast,
                                                         int planes, __nv_bfloat16* __restrict__ out) {
  __shared__ float tile[32][65];
  const int tid = threadIdx.x;
  const int64_t r0 = (int64_t)blockIdx.y * 32, k0 = (int64_t)blockIdx.x * 64, h = blockIdx.z;
  const float* base = X + h_scat[h];
  // A whole tile on regular blocks (32 rows; two 32-deep k blocks of one
  // arithmetic run): addressed from one base offset and two strides, with
  // float4 loads along a unit-stride fast index when aligned.
  int64_t rs = SCATTER_IRREGULAR, ks = SCATTER_IRREGULAR;
  if (rows_blk && k_blk && r0 + 32 <= nrows && k0 + 64 <= K) {
    rs = rows_blk[blockIdx.y];
    const int64_t k1 = k_blk[2 * blockIdx.x], k2 = k_blk[2 * blockIdx.x + 1];
    if (k1 != SCATTER_IRREGULAR && k1 == k2 && k_scat[k0 + 32] - k_scat[k0] == 32 * k1) ks = k1;
  }
  if (rs != SCATTER_IRREGULAR && ks != SCATTER_IRREGULAR) {
    const float* tb = base + rows_scat[r0] + k_scat[k0];
    const int64_t fs = kfast ? ks : rs, ss = kfast ? rs : ks;
    if (fs == 1 && (reinterpret_cast<uintptr_t>(tb) & 15) == 0 && (ss & 3) == 0) {
      // kfast: 16 threads per row (64 k); otherwise 8 threads per k column (32 rows).
      const int tpr = kfast ? 16 : 8;
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const int a0 = (tid % tpr) * 4, b = tid / tpr + j * (256 / tpr);
        const float4 v = __ldg(reinterpret_cast<const float4*>(tb + b * ss + a0));
        const float e[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          if (kfast)
            tile[b][a0 + q] = e[q];
          else
            tile[a0 + q][b] = e[q];
        }
      }
    } else {
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        int rr, kk;
        if (kfast) {
          rr = tid / 64 + 4 * j;
          kk = tid % 64;
        } else {
          rr = tid % 32;
          kk = tid / 32 + 8 * j;
        }
        tile[rr][kk] = __ldg(tb + rr * rs + kk * ks);
      }
    }
  } else {
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      int rr, kk;
      if (kfast) {
        rr = tid / 64 + 4 * j;
        kk = tid % 64;
      } else {
        rr = tid % 32;
        kk = tid / 32 + 8 * j;
      }
      const int64_t r = r0 + rr, k = k0 + kk;
      float v = 0.f;
      if (r < nrows && k < K) v = base[rows_scat[r] + k_scat[k]];
      tile[rr][kk] = v;
    }
  }
  __syncthreads();
  const int64_t plane_stride = H * rows_pad * k_pad;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int p = tid + 256 * j;
    const int rr = p / 32, kp = p % 32;
    __nv_bfloat16 a0, a1, a2, b0, b1, b2;
    split3(tile[rr][2 * kp], a0, a1, a2);
    split3(tile[rr][2 * kp + 1], b0, b1, b2);
    const int64_t off = (h * rows_pad + r0 + rr) * k_pad + k0 + 2 * kp;
    __nv_bfloat162* o = reinterpret_cast<__nv_bfloat162*>(out + off);
    o[0] = __halves2bfloat162(a0, b0);
    reinterpret_cast<__nv_bfloat162*>(out + plane_stride + off)[0] = __halves2bfloat162(a1, b1);
    if (planes > 2) reinterpret_cast<__nv_bfloat162*>(out + 2 * plane_stride + off)[0] = __halves2bfloat162(a2, b2);
  }
}

// Planes of a plain f32 or c32 operand: one 32-row x 64-deep (c32: 32 complex k)
// tile per CTA, split into three planes [H][rows_pad][k_pad], K-major. c32: A' as
// rows (re, -im) and (im, re), B' as (re, im), conjugation in the sign of im. The
// tile's largest and smallest non-zero magnitudes (as bits) go to stat.
template <bool CPLX, bool IS_A>
__global__ void __launch_bounds__(256)
plain_split_pack_kernel(const void* __restrict__ X, const int64_t* __restrict__ rows_scat,
                        const int64_t* __restrict__ k_scat, const int64_t* __restrict__ h_scat,
                        const int64_t* __restrict__ rows_blk, const int64_t* __restrict__ k_blk, int64_t nrows,
                        int64_t K, int64_t rows_pad, int64_t k_pad, int64_t H, int kfast, int conj,
                        __nv_bfloat16* __restrict__ out, uint2* __restrict__ stat) {
  using T = typename std::conditional<CPLX, float2, float>::type;
  constexpr int E = CPLX ? 2 : 1, EK = 64 / E, PR = CPLX && IS_A ? 2 : 1;
  __shared__ float tile[32][65];
  __shared__ uint2 part[8];
  const int tid = threadIdx.x;
  const int64_t r0 = (int64_t)blockIdx.y * 32, k0 = (int64_t)blockIdx.x * EK, h = blockIdx.z;
  const T* base = static_cast<const T*>(X) + h_scat[h];
  int64_t rs = SCATTER_IRREGULAR, ks = SCATTER_IRREGULAR;
  if (rows_blk && k_blk && r0 + 32 <= nrows && k0 + EK <= K) {
    rs = rows_blk[blockIdx.y];
    ks = k_blk[k0 / SCATTER_BLOCK];
    if (EK == 64 && ks != SCATTER_IRREGULAR &&
        (k_blk[k0 / SCATTER_BLOCK + 1] != ks || k_scat[k0 + 32] - k_scat[k0] != 32 * ks))
      ks = SCATTER_IRREGULAR;
  }
  const auto put = [&](int rr, int kk, T v) {
    if constexpr (CPLX) {
      tile[rr][2 * kk] = v.x;
      tile[rr][2 * kk + 1] = conj ? -v.y : v.y;
    } else {
      tile[rr][kk] = v;
    }
  };
  if (rs != SCATTER_IRREGULAR && ks != SCATTER_IRREGULAR) {
    const T* tb = base + rows_scat[r0] + k_scat[k0];
    const int64_t fs = kfast ? ks : rs, ss = kfast ? rs : ks;
    constexpr int V = 16 / (int)sizeof(T);
    if (fs == 1 && (reinterpret_cast<uintptr_t>(tb) & 15) == 0 && (ss & (V - 1)) == 0) {
      const int tpr = (kfast ? EK : 32) / V;  // threads along the fast index
#pragma unroll
      for (int j = 0; j < 32 * EK / V / 256; ++j) {
        const int a0 = (tid % tpr) * V, q = tid / tpr + j * (256 / tpr);
        const float4 x = __ldg(reinterpret_cast<const float4*>(tb + q * ss + a0));
        const T* e = reinterpret_cast<const T*>(&x);
#pragma unroll
        for (int i = 0; i < V; ++i) put(kfast ? q : a0 + i, kfast ? a0 + i : q, e[i]);
      }
    } else {
#pragma unroll
      for (int j = 0; j < 32 * EK / 256; ++j) {
        const int idx = tid + 256 * j, rr = kfast ? idx / EK : idx % 32, kk = kfast ? idx % EK : idx / 32;
        put(rr, kk, __ldg(tb + rr * rs + kk * ks));
      }
    }
  } else {
#pragma unroll
    for (int j = 0; j < 32 * EK / 256; ++j) {
      const int idx = tid + 256 * j, rr = kfast ? idx / EK : idx % 32, kk = kfast ? idx % EK : idx / 32;
      const int64_t r = r0 + rr, k = k0 + kk;
      T v{};
      if (r < nrows && k < K) v = base[rows_scat[r] + k_scat[k]];
      put(rr, kk, v);
    }
  }
  __syncthreads();
  const int64_t plane = H * rows_pad * k_pad;
  uint32_t mx = 0, mn = 0xffffffffu;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int p = tid + 256 * j, rr = p / 32, kp = p % 32;
    const float x = tile[rr][2 * kp], y = tile[rr][2 * kp + 1];
    const uint32_t bx = __float_as_uint(x) & 0x7fffffffu, by = __float_as_uint(y) & 0x7fffffffu;
    mx = max(mx, max(bx, by));
    mn = min(mn, min(bx - 1, by - 1));  // zero: the largest
    __nv_bfloat16 a[3], c[3];
    split3(x, a[0], a[1], a[2]);
    split3(y, c[0], c[1], c[2]);
    const int64_t off = (h * rows_pad + PR * (r0 + rr)) * k_pad + blockIdx.x * 64 + 2 * kp;
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      __nv_bfloat162* o = reinterpret_cast<__nv_bfloat162*>(out + q * plane + off);
      if constexpr (CPLX && IS_A) {
        if (PR * (r0 + rr) < rows_pad) {
          o[0] = __halves2bfloat162(a[q], __hneg(c[q]));
          o[k_pad / 2] = __halves2bfloat162(c[q], a[q]);
        }
      } else {
        o[0] = __halves2bfloat162(a[q], c[q]);
      }
    }
  }
  mx = __reduce_max_sync(0xffffffffu, mx);
  mn = __reduce_min_sync(0xffffffffu, mn);
  if ((tid & 31) == 0) part[tid >> 5] = make_uint2(mx, mn);
  __syncthreads();
  if (tid == 0) {
    for (int w = 1; w < 8; ++w) {
      mx = max(mx, part[w].x);
      mn = min(mn, part[w].y);
    }
    stat[(h * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x] = make_uint2(mx, mn);
  }
}

template <int S>
struct Pairs;
template <>
struct Pairs<2> {
  static constexpr int N = 3;
  __device__ static inline int a(int p) { return p == 2 ? 1 : 0; }
  __device__ static inline int b(int p) { return p == 1 ? 1 : 0; }
};
template <>
struct Pairs<3> {
  static constexpr int N = 6;
  // (0,0) (0,1) (1,0) (0,2) (1,1) (2,0)
  __device__ static inline int a(int p) { return p < 2 ? 0 : (p == 2 ? 1 : (p == 3 ? 0 : (p == 4 ? 1 : 2))); }
  __device__ static inline int b(int p) { return p == 0 ? 0 : (p == 1 ? 1 : (p == 2 ? 0 : (p == 3 ? 2 : (p == 4 ? 1 : 0)))); }
};

// split_guard of every tile from the pack's ranges: arb, brb pack rows of a tile of
// an_rb, bn_rb in all, nkb depth blocks.
__global__ void __launch_bounds__(128) split_guard_kernel(const uint2* __restrict__ sa, const uint2* __restrict__ sb,
                                                          int64_t tiles_m, int64_t tiles_n, int64_t an_rb, int64_t bn_rb,
                                                          int arb, int brb, int nkb, int k, int plain, float* __restrict__ thr,
                                                          unsigned char* __restrict__ flags) {
  int64_t h, mt, nt;
  tile_coords(blockIdx.x, tiles_m, tiles_n, h, mt, nt);
  uint32_t m[2] = {0, 0}, l[2] = {0xffffffffu, 0xffffffffu};
  const int64_t a0 = mt * arb, b0 = nt * brb;
  const int na = (int)(a0 + arb < an_rb ? arb : an_rb - a0) * nkb, nb = (int)(b0 + brb < bn_rb ? brb : bn_rb - b0) * nkb;
  for (int i = threadIdx.x; i < na; i += 128) {
    const uint2 v = sa[(h * an_rb + a0) * nkb + i];
    m[0] = max(m[0], v.x);
    l[0] = min(l[0], v.y);
  }
  for (int i = threadIdx.x; i < nb; i += 128) {
    const uint2 v = sb[(h * bn_rb + b0) * nkb + i];
    m[1] = max(m[1], v.x);
    l[1] = min(l[1], v.y);
  }
  __shared__ uint32_t part[4][4];
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    m[q] = __reduce_max_sync(0xffffffffu, m[q]);
    l[q] = __reduce_min_sync(0xffffffffu, l[q]);
    if ((threadIdx.x & 31) == 0) {
      part[threadIdx.x >> 5][q] = m[q];
      part[threadIdx.x >> 5][2 + q] = l[q];
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) {
#pragma unroll
    for (int q = 0; q < 2; ++q)
      for (int w = 1; w < 4; ++w) {
        m[q] = max(m[q], part[w][q]);
        l[q] = min(l[q], part[w][2 + q]);
      }
    const auto low = [](uint32_t x) { return x == 0xffffffffu ? 999 : (int)((x + 1) >> 23) - 127; };
    const float t = split_guard((int)(m[0] >> 23) - 127, low(l[0]), (int)(m[1] >> 23) - 127, low(l[1]), k);
    // Infinity: the whole tile is computed again; so is one with a threshold where D is
    // not only written.
    const bool whole = t == __uint_as_float(0x7f800000u) || (t != 0.f && !plain);
    thr[blockIdx.x] = whole ? __uint_as_float(0x7f800000u) : t;
    flags[blockIdx.x] = whole ? 0xff : 0;
  }
}

// 32 lanes x 64 columns, and the wait tied to its registers.
__device__ __forceinline__ void tmem_ld_x64(uint32_t taddr, uint32_t (&r)[64]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x64.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
      "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,"
      "%32,%33,%34,%35,%36,%37,%38,%39,%40,%41,%42,%43,%44,%45,%46,%47,"
      "%48,%49,%50,%51,%52,%53,%54,%55,%56,%57,%58,%59,%60,%61,%62,%63}, [%64];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), 
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), 
        "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), 
        "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31]), 
        "=r"(r[32]), "=r"(r[33]), "=r"(r[34]), "=r"(r[35]), "=r"(r[36]), "=r"(r[37]), "=r"(r[38]), "=r"(r[39]), 
        "=r"(r[40]), "=r"(r[41]), "=r"(r[42]), "=r"(r[43]), "=r"(r[44]), "=r"(r[45]), "=r"(r[46]), "=r"(r[47]), 
        "=r"(r[48]), "=r"(r[49]), "=r"(r[50]), "=r"(r[51]), "=r"(r[52]), "=r"(r[53]), "=r"(r[54]), "=r"(r[55]), 
        "=r"(r[56]), "=r"(r[57]), "=r"(r[58]), "=r"(r[59]), "=r"(r[60]), "=r"(r[61]), "=r"(r[62]), "=r"(r[63])
      : "r"(taddr));
}
__device__ __forceinline__ void tmem_wait_x64(uint32_t (&r)[64]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]), 
                 "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15]), 
                 "+r"(r[16]), "+r"(r[17]), "+r"(r[18]), "+r"(r[19]), "+r"(r[20]), "+r"(r[21]), "+r"(r[22]), "+r"(r[23]), 
                 "+r"(r[24]), "+r"(r[25]), "+r"(r[26]), "+r"(r[27]), "+r"(r[28]), "+r"(r[29]), "+r"(r[30]), "+r"(r[31]), 
                 "+r"(r[32]), "+r"(r[33]), "+r"(r[34]), "+r"(r[35]), "+r"(r[36]), "+r"(r[37]), "+r"(r[38]), "+r"(r[39]), 
                 "+r"(r[40]), "+r"(r[41]), "+r"(r[42]), "+r"(r[43]), "+r"(r[44]), "+r"(r[45]), "+r"(r[46]), "+r"(r[47]), 
                 "+r"(r[48]), "+r"(r[49]), "+r"(r[50]), "+r"(r[51]), "+r"(r[52]), "+r"(r[53]), "+r"(r[54]), "+r"(r[55]), 
                 "+r"(r[56]), "+r"(r[57]), "+r"(r[58]), "+r"(r[59]), "+r"(r[60]), "+r"(r[61]), "+r"(r[62]), "+r"(r[63])::"memory");
}

__device__ __forceinline__ void add_pair(float& x, float& y, uint32_t a, uint32_t b) {
  asm("{\n\t.reg .b64 p, q;\n\tmov.b64 p, {%0, %1};\n\tmov.b64 q, {%2, %3};\n\t"
      "add.rn.f32x2 p, p, q;\n\tmov.b64 {%0, %1}, p;\n\t}"
      : "+f"(x), "+f"(y)
      : "r"(a), "r"(b));
}

template <int S, int BN, int PLAIN = 0>
struct TcCfg {
  static constexpr int A_TILE = TC_BM * TC_BK * 2;  // bytes of one A plane tile
  static constexpr int B_TILE = BN * TC_BK * 2;
  static constexpr int STAGE = S * (A_TILE + B_TILE);
  static constexpr int STAGES = (S == 3) ? 3 : 4;
  static constexpr int RING = STAGES * STAGE;
  static constexpr int SCAT = 2 * BN * 8;  // d_n, c_n of the tile
  static constexpr int BAR = (2 * STAGES + 3) * 8 + 16;
  static constexpr int SMEM = 1024 + RING + SCAT + BAR;
  static constexpr int EPI_WARPS = 8;  // two per TMEM lane quarter, each half of the columns
  // Plain: whole warpgroups, so that the drain warps can take the registers of the others.
  static constexpr int EPI_FIRST = PLAIN ? 4 : 2;
  static constexpr int THREADS = 32 * (EPI_FIRST + EPI_WARPS);
  static constexpr int COLS_PER_THREAD = BN / 2;
};

// Two-level accumulation. The tensor core's FP32 accumulate truncates, so its
// error grows with the number of MMA steps folded into one accumulator. The
// leading product x0*y0 therefore goes into a "main" TMEM accumulator that is
// restarted every CK k-blocks; the epilogue warps drain each chunk into FP32
// registers with round-to-nearest adds. The cross terms, 2^-8 smaller, go to
// a second ("corr") accumulator that lives for the whole K loop. TMEM columns:
// main [0, BN), corr [BN, 2 BN).
//
// Tail split: the grid is 1-D; CTAs [0, whole) own one tile each over all of
// K, and the last `tail` tiles (those that would run as a partly filled last
// wave) are split into `parts` K ranges of whole CK chunks, one CTA each. A
// tail CTA writes its FP32 sum to partial[(tail tile * parts + part) * TC_BM
// * BN + col * TC_BM + row] and split_tail_reduce_kernel adds the parts in
// order and applies the epilogue.
//
// PLAIN 0: the split schemes; 1 and 2: plain f32 and c32, with the tiles' thresholds.
// There the main accumulator restarts every 16-deep step: 16 16-bit products mostly add
// up exactly, so values of one sign gather no bias from the truncation (x1 y2, x2 y1 and
// x2 y2 are left out, up to 2^-24 of a product and 2^-26 typically; with all of them the
// error is the same from K = 512 on). The cross terms of a step cover the drain of the
// one before; the drain warps take the registers of the other roles and release the
// accumulator before they add. The FP32 sums of 16 or 32 steps go to a second sum per
// output (in local memory, an eighth of the columns at a time), so that the roundings
// of a long K do not pile up. f32 4096^3 on B200: 626 us with restarts every 64 k and
// one sum, 775 so (731 without the second sum); error on uniform [0, 1) 1.3e-7 -> 0.6e-7
// (FFMA tiles 1.1e-7), on [-1, 1) 1.7e-7 -> 1.25e-7 (2.1e-7).
template <int S, int BN, int CK, int PLAIN>
__global__ void __launch_bounds__(TcCfg<S, BN, PLAIN>::THREADS, 1)
tc_bf16_gemm_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, GemmArgs g,
                    int64_t m_pad, int64_t n_pad, int64_t k_pad, int64_t whole, int parts, float* partial,
                    const float* __restrict__ thr_of, unsigned char* __restrict__ flags) {
  using Cfg = TcCfg<S, BN, PLAIN>;
  constexpr int CPT = Cfg::COLS_PER_THREAD;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* ring = smem;
  int64_t* dn_s = reinterpret_cast<int64_t*>(smem + Cfg::RING);
  int64_t* cn_s = dn_s + BN;
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + Cfg::RING + Cfg::SCAT);
  uint64_t* empty = full + Cfg::STAGES;
  uint64_t* main_full = empty + Cfg::STAGES;
  uint64_t* main_empty = main_full + 1;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(main_empty + 1);

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int64_t tiles_n = n_pad / BN, tiles_m = m_pad / TC_BM;
  const int nk_all = (int)(k_pad / TC_BK);
  int64_t tile = blockIdx.x;
  int part = -1;  // -1: the whole K range
  int kb_lo = 0, kb_hi = nk_all;
  if ((int64_t)blockIdx.x >= whole) {
    const int64_t j = (int64_t)blockIdx.x - whole;
    tile = whole + j / parts;
    part = (int)(j % parts);
    const int per = ((nk_all + parts - 1) / parts + CK - 1) / CK * CK;  // whole chunks per part
    kb_lo = part * per;
    kb_hi = kb_lo + per < nk_all ? kb_lo + per : nk_all;
  }
  int64_t h, mt, nt;
  tile_coords(tile, tiles_m, tiles_n, h, mt, nt);
  const int64_t m0 = mt * TC_BM, n0 = nt * BN;
  // Sums below thr may have lost bits; infinity: the tile is computed by FFMA (k_again.cu).
  const float thr = PLAIN ? thr_of[tile] : 0.f;
  const bool whole_tile = PLAIN != 0 && thr == __uint_as_float(0x7f800000u);
  const int nk = whole_tile ? 0 : kb_hi - kb_lo;  // k-blocks of this CTA
  const int nchunks = (nk + CK - 1) / CK;

  if (warp == 0 && lane == 0) {
    for (int i = 0; i < Cfg::STAGES; ++i) {
      mbar_init(&full[i], 1);
      mbar_init(&empty[i], 1);
    }
    mbar_init(main_full, 1);
    mbar_init(main_empty, Cfg::EPI_WARPS);
    fence_barrier_init();
    asm volatile("prefetch.tensormap [%0];" ::"l"(&tmA) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&tmB) : "memory");
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, 2 * BN);
    tmem_relinquish();
  }
  if (warp >= Cfg::EPI_FIRST) {
    for (int i = tid - 32 * Cfg::EPI_FIRST; i < BN; i += 32 * Cfg::EPI_WARPS) {
      const int64_t n = n0 + i;
      const bool ok = n < g.N;
      dn_s[i] = ok ? g.s.d_n[n] : 0;
      cn_s[i] = ok ? g.s.c_n[n] : 0;
    }
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  const uint32_t tmem_main = tmem, tmem_corr = tmem + BN;

  // Plain: registers a thread 40 x 128 + 232 x 256 = 64512 of the launch's 168 x 384.
  if (warp < Cfg::EPI_FIRST) {
    if constexpr (PLAIN != 0) asm volatile("setmaxnreg.dec.sync.aligned.u32 40;");
    if (warp == 0) {
      if (lane == 0) {
        for (int kb = 0; kb < nk; ++kb) {
          const int st = kb % Cfg::STAGES;
          const uint32_t round = (uint32_t)(kb / Cfg::STAGES);
          if (!mbar_wait(&empty[st], (round & 1u) ^ 1u)) {
            atomicOr(g.status, STATUS_WAIT_TIMEOUT);
            break;
          }
          mbar_arrive_expect_tx(&full[st], (uint32_t)Cfg::STAGE);
          uint8_t* sbase = ring + st * Cfg::STAGE;
          const int kx = (kb_lo + kb) * TC_BK;
#pragma unroll
          for (int p = 0; p < S; ++p)
            tma_load_2d(sbase + p * Cfg::A_TILE, &tmA, &full[st], kx, (int)((p * g.H + h) * m_pad + m0));
#pragma unroll
          for (int p = 0; p < S; ++p)
            tma_load_2d(sbase + S * Cfg::A_TILE + p * Cfg::B_TILE, &tmB, &full[st], kx,
                        (int)((p * g.H + h) * n_pad + n0));
        }
      }
    } else if (warp == 1) {
      if (lane == 0) {
        constexpr uint32_t IDESC = idesc_bf16(TC_BM, BN);
        bool ok = true;
        for (int kb = 0; kb < nk && ok; ++kb) {
          const int st = kb % Cfg::STAGES;
          const uint32_t round = (uint32_t)(kb / Cfg::STAGES);
          if (!mbar_wait(&full[st], round & 1u)) {
            atomicOr(g.status, STATUS_WAIT_TIMEOUT);
            break;
          }
          tc_fence_after();
          const uint32_t sbase = smem_u32(ring + st * Cfg::STAGE);
          if constexpr (PLAIN != 0) {
#pragma unroll
            for (int kk = 0; kk < 2; ++kk) {
              uint64_t a[3], b[3];
#pragma unroll
              for (int p = 0; p < 3; ++p) {
                a[p] = sdesc_sw64(sbase + p * Cfg::A_TILE) + 2 * kk;
                b[p] = sdesc_sw64(sbase + S * Cfg::A_TILE + p * Cfg::B_TILE) + 2 * kk;
              }
              umma_bf16(tmem_corr, a[0], b[2], IDESC, (kb | kk) != 0 ? 1u : 0u);
              umma_bf16(tmem_corr, a[2], b[0], IDESC, 1u);
              umma_bf16(tmem_corr, a[1], b[1], IDESC, 1u);
              umma_bf16(tmem_corr, a[0], b[1], IDESC, 1u);
              umma_bf16(tmem_corr, a[1], b[0], IDESC, 1u);
              if (!mbar_wait_polls(main_empty, (uint32_t)kk ^ 1u)) {
                atomicOr(g.status, STATUS_WAIT_TIMEOUT);
                ok = false;
                break;
              }
              tc_fence_after();
              umma_bf16(tmem_main, a[0], b[0], IDESC, 0u);
              umma_commit(main_full);
            }
            umma_commit(&empty[st]);
          } else {
            // Cross terms first: they overlap the drain of the previous chunk.
#pragma unroll
            for (int p = 1; p < Pairs<S>::N; ++p) {
              const uint64_t ad = sdesc_sw64(sbase + Pairs<S>::a(p) * Cfg::A_TILE);
              const uint64_t bd = sdesc_sw64(sbase + S * Cfg::A_TILE + Pairs<S>::b(p) * Cfg::B_TILE);
#pragma unroll
              for (int kk = 0; kk < TC_BK / 16; ++kk)
                umma_bf16(tmem_corr, ad + 2 * kk, bd + 2 * kk, IDESC, (kb | (p - 1) | kk) != 0 ? 1u : 0u);
            }
            const int chunk = kb / CK, in_chunk = kb % CK;
            if (in_chunk == 0 && !mbar_wait(main_empty, ((uint32_t)chunk & 1u) ^ 1u)) {
              atomicOr(g.status, STATUS_WAIT_TIMEOUT);
              ok = false;
            }
            tc_fence_after();
            {
              const uint64_t ad = sdesc_sw64(sbase);
              const uint64_t bd = sdesc_sw64(sbase + S * Cfg::A_TILE);
#pragma unroll
              for (int kk = 0; kk < TC_BK / 16; ++kk)
                umma_bf16(tmem_main, ad + 2 * kk, bd + 2 * kk, IDESC, (in_chunk | kk) != 0 ? 1u : 0u);
            }
            umma_commit(&empty[st]);
            if (in_chunk == CK - 1 || kb == nk - 1) umma_commit(main_full);
          }
        }
        if (PLAIN == 0 && !ok) umma_commit(main_full);
      }
    }
  } else {
    if constexpr (PLAIN != 0) asm volatile("setmaxnreg.inc.sync.aligned.u32 232;");
    // Epilogue: warp w reads TMEM lanes 32*(w%4) .. +31 (tile rows) and half
    // of the columns; it keeps the running FP32 sum of its 128 outputs.
    const int lane_base = 32 * (warp & 3);
    const int col0 = ((warp - Cfg::EPI_FIRST) >> 2) * CPT;
    const uint32_t lane_addr = (uint32_t)lane_base << 16;
    float run[CPT];
#pragma unroll
    for (int j = 0; j < CPT; ++j) run[j] = 0.f;
    bool ok = true;
    if constexpr (PLAIN != 0) {
      constexpr int GROUPS = CPT / 16;
      const int every = nk > 32 ? 4 : 2;  // steps per group of columns whose sums move
      __align__(16) float kept[CPT];
      float* sums = kept;
      asm volatile("" : "+l"(sums));  // in local memory
      for (int c = 0; c < 2 * nk; ++c) {
        // The group whose sums move after this step, fetched ahead of the wait.
        const int group = c % every == every - 1 ? c / every % GROUPS : -1;
        float p[16];
        if (group >= 0 && c >= every * GROUPS) {
#pragma unroll
          for (int j = 0; j < 16; j += 4) *reinterpret_cast<float4*>(p + j) = *reinterpret_cast<float4*>(sums + 16 * group + j);
        } else {
#pragma unroll
          for (int j = 0; j < 16; ++j) p[j] = 0.f;
        }
        if (!mbar_wait_polls(main_full, (uint32_t)c & 1u)) {
          atomicOr(g.status, STATUS_WAIT_TIMEOUT);
          ok = false;
          break;
        }
        tc_fence_after();
#pragma unroll
        for (int q = 0; q < CPT / 64; ++q) {
          uint32_t r[64];
          tmem_ld_x64(tmem_main + lane_addr + (uint32_t)(col0 + 64 * q), r);
          tmem_wait_x64(r);
          if (q == CPT / 64 - 1) {  // read: the next step may fill it again
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(main_empty);
          }
#pragma unroll
          for (int j = 0; j < 64; j += 2) add_pair(run[64 * q + j], run[64 * q + j + 1], r[j], r[j + 1]);
        }
#pragma unroll
        for (int q = 0; q < GROUPS; ++q)
          if (group == q) {
#pragma unroll
            for (int j = 0; j < 16; j += 4) {
              *reinterpret_cast<float4*>(sums + 16 * q + j) =
                  make_float4(p[j] + run[16 * q + j], p[j + 1] + run[16 * q + j + 1], p[j + 2] + run[16 * q + j + 2],
                              p[j + 3] + run[16 * q + j + 3]);
              run[16 * q + j] = run[16 * q + j + 1] = run[16 * q + j + 2] = run[16 * q + j + 3] = 0.f;
            }
          }
      }
#pragma unroll
      for (int q = 0; q < GROUPS; ++q)
        if (2 * nk >= every * (q + 1)) {
#pragma unroll
          for (int j = 0; j < 16; ++j) run[16 * q + j] += sums[16 * q + j];
        }
    }
    for (int c = 0; PLAIN == 0 && c < nchunks; ++c) {
      if (!mbar_wait(main_full, (uint32_t)c & 1u)) {
        atomicOr(g.status, STATUS_WAIT_TIMEOUT);
        ok = false;
        break;
      }
      tc_fence_after();
#pragma unroll
      for (int q = 0; q < CPT / 16; ++q) {
        uint32_t r[16];
        tmem_ld_32x32b_x16(tmem_main + lane_addr + (uint32_t)(col0 + 16 * q), r);
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 16; ++j) run[16 * q + j] += __uint_as_float(r[j]);
      }
      tc_fence_before();
      if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(main_empty)) : "memory");
    }
    constexpr bool CPLX = PLAIN == 2;
    const int64_t m = CPLX ? (m0 + lane_base + lane) >> 1 : m0 + lane_base + lane;
    const bool mok = ok && m < g.M;
    const int64_t dm = mok ? g.s.d_m[m] : 0;
    const int64_t cm = (mok && !g.e.beta_zero) ? g.s.c_m[m] : 0;
    using T = typename Elem<float, CPLX>::type;
    const T* Cb = static_cast<const T*>(g.C) + (g.e.beta_zero ? 0 : g.s.h_c[h]) + cm;
    T* Db = static_cast<T*>(g.D) + g.s.h_d[h] + dm;
    float least = __uint_as_float(0x7f800000u);  // magnitude of what this lane writes
    float* Pb = part >= 0 ? partial + ((tile - whole) * parts + part) * (int64_t)(TC_BM * BN) + lane_base + lane
                          : nullptr;
    // The last main_full commit also covers every cross-term MMA.
#pragma unroll
    for (int q = 0; q < (whole_tile ? 0 : CPT / 16); ++q) {
      uint32_t r[16];
      tmem_ld_32x32b_x16(tmem_corr + lane_addr + (uint32_t)(col0 + 16 * q), r);
      tmem_ld_wait(r);
      if (part >= 0) {
        // Tail part: the raw FP32 sum, column-major in the tile (coalesced).
#pragma unroll
        for (int j = 0; j < 16; ++j) Pb[(col0 + 16 * q + j) * TC_BM] = run[16 * q + j] + __uint_as_float(r[j]);
      } else if constexpr (PLAIN != 0) {
        const int comp = CPLX ? lane & 1 : 0;
        constexpr int CG = CPLX ? 4 : 8;
        if (thr != 0.f) {
#pragma unroll
          for (int j = 0; j < 16; ++j)
            if (n0 + col0 + 16 * q + j < g.N) least = fminf(least, fabsf(run[16 * q + j] + __uint_as_float(r[j])));
        }
        if (g.e.plain) {
          if (mok) {
#pragma unroll
            for (int j = 0; j < 16; ++j) {
              const int nn = col0 + 16 * q + j;
              if (n0 + nn < g.N)
                reinterpret_cast<float*>(Db + dn_s[nn])[comp] = run[16 * q + j] + __uint_as_float(r[j]);
            }
          }
          __syncwarp();
          continue;
        }
#pragma unroll
        for (int j0 = 0; j0 < 16; j0 += CG) {
          T cv[CG];  // C of the group, on its way before the first of it is used
          if (!g.e.beta_zero) {
#pragma unroll
            for (int j = 0; j < CG; ++j)
              if (mok && n0 + col0 + 16 * q + j0 + j < g.N && !comp) cv[j] = Cb[cn_s[col0 + 16 * q + j0 + j]];
          }
#pragma unroll
          for (int j = 0; j < CG; ++j) {
            const int jj = 16 * q + j0 + j, nn = col0 + jj;
            const float v = run[jj] + __uint_as_float(r[j0 + j]);
            const float o = CPLX ? __shfl_xor_sync(0xffffffffu, v, 1) : 0.f;
            if (mok && n0 + nn < g.N && !comp) epilogue_store<float, CPLX>(g.e, v, o, &cv[j], Db + dn_s[nn]);
          }
        }
      } else if (mok) {
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          const int nn = col0 + 16 * q + j;
          if (n0 + nn < g.N)
            epilogue_store<float, CPLX>(g.e, run[16 * q + j] + __uint_as_float(r[j]), 0.f, Cb + cn_s[nn],
                                        Db + dn_s[nn]);
        }
      }
    }
    if (PLAIN != 0 && part < 0 && thr != 0.f && __any_sync(0xffffffffu, mok && !(least >= thr)) && lane == 0)
      mark_again(flags, tile, warp - Cfg::EPI_FIRST);
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem, 2 * BN);
  }
}

// Tail tiles: add the parts in order, then the epilogue through the scatter.
template <int BN>
__global__ void __launch_bounds__(256) split_tail_reduce_kernel(GemmArgs g, const float* __restrict__ partial,
                                                                int64_t whole, int parts, int64_t tail, int64_t m_pad,
                                                                int64_t n_pad) {
  const int64_t tiles_n = n_pad / BN, tiles_m = m_pad / TC_BM;
  const int64_t total = tail * TC_BM * BN;
  for (int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; idx < total;
       idx += (int64_t)gridDim.x * blockDim.x) {
    const int64_t t = idx / (TC_BM * BN), within = idx % (TC_BM * BN);
    const int row = (int)(within % TC_BM), col = (int)(within / TC_BM);
    const int64_t tile = whole + t;
    int64_t h, mt, nt;
    tile_coords(tile, tiles_m, tiles_n, h, mt, nt);
    const int64_t m = mt * TC_BM + row, n = nt * BN + col;
    if (m >= g.M || n >= g.N) continue;
    float v = 0.f;
    for (int p = 0; p < parts; ++p) v += partial[(t * parts + p) * (int64_t)(TC_BM * BN) + within];
    const float* c = static_cast<const float*>(g.C) + (g.e.beta_zero ? 0 : g.s.h_c[h] + g.s.c_m[m] + g.s.c_n[n]);
    float* d = static_cast<float*>(g.D) + g.s.h_d[h] + g.s.d_m[m] + g.s.d_n[n];
    epilogue_store<float, false>(g.e, v, 0.f, c, d);
  }
}

// The same for plain f32 and c32, whose sums below the tile's threshold are marked.
template <int BN, bool CPLX>
__global__ void __launch_bounds__(256) plain_tail_reduce_kernel(GemmArgs g, const float* __restrict__ partial,
                                                                int64_t whole, int parts, int64_t tail, int64_t m_pad,
                                                                int64_t n_pad, const float* __restrict__ thr_of,
                                                                unsigned char* __restrict__ flags) {
  using T = typename Elem<float, CPLX>::type;
  const int64_t tiles_n = n_pad / BN, tiles_m = m_pad / TC_BM;
  const int64_t total = tail * TC_BM * BN;
  for (int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; idx < total;
       idx += (int64_t)gridDim.x * blockDim.x) {
    const int64_t t = idx / (TC_BM * BN), within = idx % (TC_BM * BN);
    const int row = (int)(within % TC_BM), col = (int)(within / TC_BM);
    const int64_t tile = whole + t;
    int64_t h, mt, nt;
    tile_coords(tile, tiles_m, tiles_n, h, mt, nt);
    const int64_t m = CPLX ? (mt * TC_BM + row) >> 1 : mt * TC_BM + row, n = nt * BN + col;
    if (m >= g.M || n >= g.N || (CPLX && (row & 1))) continue;
    const float thr = thr_of[tile];
    if (thr == __uint_as_float(0x7f800000u)) continue;
    float v = 0.f, o = 0.f;
    for (int p = 0; p < parts; ++p) {
      v += partial[(t * parts + p) * (int64_t)(TC_BM * BN) + within];
      if (CPLX) o += partial[(t * parts + p) * (int64_t)(TC_BM * BN) + within + 1];
    }
    if (thr != 0.f && !(fabsf(v) >= thr && (!CPLX || fabsf(o) >= thr))) mark_again(flags, tile, row / 32 + 4 * (col / (BN / 2)));
    const T* c = static_cast<const T*>(g.C) + (g.e.beta_zero ? 0 : g.s.h_c[h] + g.s.c_m[m] + g.s.c_n[n]);
    T* d = static_cast<T*>(g.D) + g.s.h_d[h] + g.s.d_m[m] + g.s.d_n[n];
    epilogue_store<float, CPLX>(g.e, v, o, c, d);
  }
}

// The tail split for a grid of `tiles` tiles on `sms` SMs (one CTA per SM):
// the tiles of a partly filled last wave are split into `parts` K ranges when
// that fills the wave better; parts = 1 means no split.
struct TailSplit {
  int64_t whole, tail;
  int parts;
};
// `deep`: also a first wave that is partly filled (up to 16 parts).
inline TailSplit tail_split(int64_t tiles, int sms, int nk, int ck, bool deep = false) {
  TailSplit t{tiles, 0, 1};
  const int64_t rem = tiles % sms;
  if (rem == 0 || (tiles < sms && !deep)) return t;  // full waves, or one partial wave of whole tiles
  int parts = (int)(sms / rem);
  const int most = tiles < sms ? 16 : 4;
  parts = parts < most ? parts : most;
  // Each part keeps at least two CK chunks and the last part is not empty.
  auto fits = [&](int p) {
    const int per = ((nk + p - 1) / p + ck - 1) / ck * ck;
    return nk >= p * 2 * ck && (p - 1) * per < nk;
  };
  while (parts > 1 && !fits(parts)) --parts;
  if (parts < 2) return t;
  t.whole = tiles - rem;
  t.tail = rem;
  t.parts = parts;
  return t;
}

constexpr int TC_PLAIN_SMS = 148;  // what the plain path's workspace is sized for

template <int S, int BN, int CK, int PLAIN = 0>
cudaError_t run_tc(const GemmArgs& g, const SplitLayout& L, const void* ap, const void* bp, float* tail_partial,
                   cudaStream_t st, const float* thr = nullptr, unsigned char* flags = nullptr) {
  using Cfg = TcCfg<S, BN, PLAIN>;
  CUtensorMap ma, mb;
  if (!make_map_2d(&ma, ap, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, L.k_pad, (int64_t)S * L.H * L.m_pad, TC_BK, TC_BM))
    return cudaErrorInvalidValue;
  if (!make_map_2d(&mb, bp, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, L.k_pad, (int64_t)S * L.H * L.n_pad, TC_BK, BN))
    return cudaErrorInvalidValue;
  // Per call: the attribute belongs to the current device's context.
  cudaError_t e =
      cudaFuncSetAttribute(tc_bf16_gemm_kernel<S, BN, CK, PLAIN>, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::SMEM);
  if (e != cudaSuccess) return e;
  const int64_t tiles = (L.n_pad / BN) * (L.m_pad / TC_BM) * L.H;
  TailSplit ts{tiles, 0, 1};
  if (tail_partial) {
    int dev = 0, sms = 148;
    if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (PLAIN && sms > TC_PLAIN_SMS) sms = TC_PLAIN_SMS;
    ts = tail_split(tiles, sms, (int)(L.k_pad / TC_BK), CK, PLAIN != 0);
  }
  const int64_t grid = ts.whole + ts.tail * ts.parts;
  tc_bf16_gemm_kernel<S, BN, CK, PLAIN><<<(unsigned)grid, Cfg::THREADS, Cfg::SMEM, st>>>(
      ma, mb, g, L.m_pad, L.n_pad, L.k_pad, ts.whole, ts.parts, tail_partial, thr, flags);
  e = cudaGetLastError();
  if (e != cudaSuccess || ts.tail == 0) return e;
  const int64_t elems = ts.tail * TC_BM * BN;
  const unsigned blocks = (unsigned)((elems + 255) / 256 < 4096 ? (elems + 255) / 256 : 4096);
  if constexpr (PLAIN != 0)
    plain_tail_reduce_kernel<BN, PLAIN == 2><<<blocks, 256, 0, st>>>(g, tail_partial, ts.whole, ts.parts, ts.tail, L.m_pad,
                                                                     L.n_pad, thr, flags);
  else
    split_tail_reduce_kernel<BN><<<blocks, 256, 0, st>>>(g, tail_partial, ts.whole, ts.parts, ts.tail, L.m_pad, L.n_pad);
  return cudaGetLastError();
}

}  // namespace

SplitLayout split_layout(int scheme, int64_t M, int64_t N, int64_t K, int64_t H) {
  SplitLayout L;
  L.planes = (scheme == 2) ? 3 : 2;
  L.m_pad = (M + TC_BM - 1) / TC_BM * TC_BM;
  L.n_pad = (N + 255) / 256 * 256;
  L.k_pad = (K + 63) / 64 * 64;
  L.H = H;
  return L;
}

size_t split_workspace_bytes(const SplitLayout& L) {
  return (size_t)L.planes * (size_t)L.H * (size_t)(L.m_pad + L.n_pad) * (size_t)L.k_pad * 2 + 256;
}

cudaError_t launch_split_pack_f32(const GemmArgs& g, int which, const SplitLayout& L, void* planes, cudaStream_t st) {
  const bool a = which == 0;
  const int64_t rows_pad = a ? L.m_pad : L.n_pad;
  dim3 grid((unsigned)(L.k_pad / 64), (unsigned)(rows_pad / 32), (unsigned)L.H);
  if (L.H > 65535 || rows_pad / 32 > 65535) return cudaErrorInvalidConfiguration;
  split_pack_kernel<<<grid, 256, 0, st>>>(static_cast<const float*>(a ? g.A : g.B), a ? g.s.a_m : g.s.b_n,
                                          a ? g.s.a_k : g.s.b_k, a ? g.s.h_a : g.s.h_b, a ? g.s.blk_a_m : g.s.blk_b_n,
                                          a ? g.s.blk_a_k : g.s.blk_b_k, a ? g.M : g.N, g.K, rows_pad,
                                          L.k_pad, L.H, a ? g.a_kfast : g.b_kfast, L.planes,
                                          static_cast<__nv_bfloat16*>(planes));
  return cudaGetLastError();
}

int split_tail_parts(const SplitLayout& L, int num_sms) {
  const int64_t tiles = (L.n_pad / 256) * (L.m_pad / TC_BM) * L.H;
  return tail_split(tiles, num_sms, (int)(L.k_pad / TC_BK), 4).parts;
}

size_t split_tail_bytes(const SplitLayout& L, int num_sms) {
  // At most one wave of tail parts (tail * parts <= num_sms) of 128 x 256 FP32.
  (void)L;
  return (size_t)num_sms * TC_BM * 256 * sizeof(float) + 256;
}

cudaError_t launch_tc_bf16_gemm(const GemmArgs& g, const SplitLayout& L, const void* ap, const void* bp, int scheme,
                                cudaStream_t st, void* tail_partial) {
  if ((int64_t)L.planes * L.H * (L.m_pad > L.n_pad ? L.m_pad : L.n_pad) >= (int64_t)1 << 31)
    return cudaErrorInvalidValue;
  if (L.H > 65535) return cudaErrorInvalidConfiguration;
  float* tp = static_cast<float*>(tail_partial);
  if (scheme == 2) return run_tc<3, 256, 4>(g, L, ap, bp, tp, st);
  return run_tc<2, 256, 4>(g, L, ap, bp, tp, st);
}

// ---- plain f32 / c32 --------------------------------------------------------

namespace {
// The workspace: A' planes, B' planes, their ranges, the tiles' thresholds and flags,
// the tail parts.
struct PlainSplitSpace {
  size_t b, sa, sb, thr, flags, tail, bytes;
  int64_t a_rb, b_rb, nkb;
};
PlainSplitSpace plain_split_space(int dtype, const SplitLayout& L) {
  const auto up = [](size_t x) { return (x + 255) & ~size_t(255); };
  PlainSplitSpace s;
  s.a_rb = L.m_pad / (dtype == 2 ? 64 : 32);
  s.b_rb = L.n_pad / 32;
  s.nkb = L.k_pad / 64;
  s.b = up((size_t)3 * L.H * L.m_pad * L.k_pad * 2);
  s.sa = s.b + up((size_t)3 * L.H * L.n_pad * L.k_pad * 2);
  s.sb = s.sa + up((size_t)L.H * s.a_rb * s.nkb * 8);
  s.thr = s.sb + up((size_t)L.H * s.b_rb * s.nkb * 8);
  const size_t tiles = (size_t)(L.m_pad / TC_BM) * (L.n_pad / 256) * L.H;
  s.flags = s.thr + up(tiles * 4);
  s.tail = s.flags + up(tiles);
  s.bytes = s.tail + up(split_tail_bytes(L, TC_PLAIN_SMS));
  return s;
}
}  // namespace

bool is_tc_split(int kernel) { return kernel == PLAIN_F32_TC_SPLIT || kernel == PLAIN_C32_TC_SPLIT; }

SplitLayout plain_split_layout(int dtype, int64_t M, int64_t N, int64_t K, int64_t H) {
  return split_layout(2, dtype == 2 ? 2 * M : M, N, dtype == 2 ? 2 * K : K, H);
}
size_t plain_split_bytes(int dtype, int64_t M, int64_t N, int64_t K, int64_t H) {
  const SplitLayout a = plain_split_layout(dtype, M, N, K, H), b = plain_split_layout(dtype, N, M, K, H);
  const size_t x = plain_split_space(dtype, a).bytes, y = plain_split_space(dtype, b).bytes;
  return (x > y ? x : y) + 256;  // either orientation
}

bool tc_split_fits(int dtype, int64_t M, int64_t N, int64_t K, int64_t H) {
  if ((dtype != 0 && dtype != 2) || K <= 0 || H > 65535) return false;
  const int64_t most = (int64_t)1 << 30;
  if (M >= most / 8 || N >= most / 8 || K >= most / 8) return false;
  const int64_t rows = (M > N ? M : N) * 2 + 256;
  return rows / 32 <= 65535 && 3 * H * rows < 2 * most && (M / 64 + 2) * (N / 64 + 2) * H < most;
}

cudaError_t launch_plain_split_pack(int dtype, const GemmArgs& g, int which, void* ws, cudaStream_t st) {
  const SplitLayout L = plain_split_layout(dtype, g.M, g.N, g.K, g.H);
  const PlainSplitSpace S = plain_split_space(dtype, L);
  char* w = static_cast<char*>(ws);
  const bool a = which == 0;
  const dim3 grid((unsigned)S.nkb, (unsigned)(a ? S.a_rb : S.b_rb), (unsigned)L.H);
  auto kern = dtype == 2 ? (a ? plain_split_pack_kernel<true, true> : plain_split_pack_kernel<true, false>)
                         : (a ? plain_split_pack_kernel<false, true> : plain_split_pack_kernel<false, false>);
  kern<<<grid, 256, 0, st>>>(a ? g.A : g.B, a ? g.s.a_m : g.s.b_n, a ? g.s.a_k : g.s.b_k, a ? g.s.h_a : g.s.h_b,
                             a ? g.s.blk_a_m : g.s.blk_b_n, a ? g.s.blk_a_k : g.s.blk_b_k, a ? g.M : g.N, g.K,
                             a ? L.m_pad : L.n_pad, L.k_pad, L.H, a ? g.a_kfast : g.b_kfast, a ? g.conj_a : g.conj_b,
                             reinterpret_cast<__nv_bfloat16*>(a ? w : w + S.b),
                             reinterpret_cast<uint2*>(w + (a ? S.sa : S.sb)));
  return cudaGetLastError();
}

cudaError_t launch_plain_split_gemm(int dtype, const GemmArgs& g, void* ws, cudaStream_t st) {
  const SplitLayout L = plain_split_layout(dtype, g.M, g.N, g.K, g.H);
  const PlainSplitSpace S = plain_split_space(dtype, L);
  char* w = static_cast<char*>(ws);
  const int64_t tm = L.m_pad / TC_BM, tn = L.n_pad / 256;
  float* thr = reinterpret_cast<float*>(w + S.thr);
  unsigned char* flags = reinterpret_cast<unsigned char*>(w + S.flags);
  split_guard_kernel<<<(unsigned)(tm * tn * L.H), 128, 0, st>>>(
      reinterpret_cast<const uint2*>(w + S.sa), reinterpret_cast<const uint2*>(w + S.sb), tm, tn, S.a_rb, S.b_rb,
      dtype == 2 ? 2 : 4, 8, (int)S.nkb, (int)L.k_pad, g.e.plain, thr, flags);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  float* tail = reinterpret_cast<float*>(w + S.tail);
  e = dtype == 2 ? run_tc<3, 256, 1, 2>(g, L, w, w + S.b, tail, st, thr, flags)
                 : run_tc<3, 256, 1, 1>(g, L, w, w + S.b, tail, st, thr, flags);
  if (e != cudaSuccess) return e;
  return launch_ffma_again(dtype, g, flags, tm * tn * L.H, tm, tn, 256, true, TC_PLAIN_SMS, st);
}

}  // namespace dev
}  // namespace tprims
