// Batches of small products (M, N, K <= 32): whole products in shared memory.
//
// Such a batch is bound by HBM: every operand element is used a few dozen times
// at most, so a tile of a product is one round of loads, a short product and one
// round of stores. A CTA takes G consecutive batch entries, copies their A' and
// B' into shared memory element by element with cp.async in the operand's own
// memory order (batch, row and depth index sorted by stride, so that neighbouring
// lanes read neighbouring elements whichever index is innermost), forms every
// output of the group in registers (T x T outputs a thread, one thread per output
// block, K in order), and writes D through shared memory in D's own memory order.
// A side whose batch entries follow one another in memory moves in 16-byte copies
// (D in 16-byte stores) and keeps the memory's order in shared memory. About 36 KB
// of shared memory per CTA keeps six CTAs, and their loads, in flight per SM (24 KB
// measured 2 to 19 % slower). f64 8192 products of 32 x 4 x 32 on B200: 123 us on
// 64 x 64 tiles, 16.4 us here in calls one after another (84 MB, 5.1 TB/s).
#include "device_common.cuh"

namespace tprims {
namespace dev {

namespace {

constexpr int SB_NT = 128;
constexpr int SB_SMEM = 36 * 1024;  // per CTA, one product alone may take more

// One operand (or D, C): its three indexes (batch, row, depth or column) from
// the smallest stride to the largest.
struct SmallSide {
  int size[3];            // extents; the batch one is the group size
  int dst[3];             // element strides in shared memory
  int64_t st[3];          // element strides (regular layouts)
  const int64_t* vec[3];  // offsets (other layouts)
  int hdim;               // which of the three is the batch
  int linear;             // the group's elements are one contiguous run, kept in that order
};

struct SmallArgs {
  SmallSide a, b, d, c;  // c: in d's index order
  int G, mt, nt;         // entries per CTA; row and column blocks of a product
  // Shared-memory strides (elements) of an entry, its rows (columns) and depth.
  int as, ar, ak, bs, bn, bk, ds, dr, dc;
  int b_off;  // byte offset of B'
  int wide;   // element copies of the whole element (operands aligned to it)
};

template <int BYTES>
__device__ __forceinline__ void small_copy(void* smem, const void* gmem) {
  const uint32_t s = (uint32_t)__cvta_generic_to_shared(smem);
  if constexpr (BYTES == 16)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(s), "l"(gmem) : "memory");
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(s), "l"(gmem), "n"(BYTES) : "memory");
}

// Visits the elements of a side in memory order, f(index offset of the element,
// shared-memory index, i0, i1, i2); `gcount` entries of the group exist.
template <bool REG, class F>
__device__ __forceinline__ void small_visit(const SmallSide& s, int64_t h0, int gcount, F&& f) {
  const int n0 = s.hdim == 0 ? gcount : s.size[0], n1 = s.hdim == 1 ? gcount : s.size[1],
            n2 = s.hdim == 2 ? gcount : s.size[2];
  const int total = n0 * n1 * n2, t = threadIdx.x;
  // Indexes advance by SB_NT elements a step: carries instead of divisions.
  int i0 = t % n0, r = t / n0, i1 = r % n1, i2 = r / n1;
  const int d0 = SB_NT % n0, rr = SB_NT / n0, d1 = rr % n1, d2 = rr / n1;
  for (int e = t; e < total; e += SB_NT) {
    int64_t off;
    if (REG) {
      off = i0 * s.st[0] + i1 * s.st[1] + i2 * s.st[2] + h0 * s.st[s.hdim];
    } else {
      off = s.vec[0][i0 + (s.hdim == 0 ? h0 : 0)] + s.vec[1][i1 + (s.hdim == 1 ? h0 : 0)] +
            s.vec[2][i2 + (s.hdim == 2 ? h0 : 0)];
    }
    f(off, i0 * s.dst[0] + i1 * s.dst[1] + i2 * s.dst[2], i0, i1, i2);
    i0 += d0;
    i1 += d1;
    i2 += d2;
    if (i0 >= n0) {
      i0 -= n0;
      ++i1;
    }
    if (i1 >= n1) {
      i1 -= n1;
      ++i2;
    }
  }
}

// Copies the group of a linear side to shared memory at the source's own offset
// within 16 bytes (returned): 16-byte copies, single elements at both ends.
template <class E, int UNIT>
__device__ __forceinline__ int small_linear(const SmallSide& s, const E* src, char* dst, int64_t h0, int gcount) {
  const int n = gcount * s.size[0] * s.size[1];  // hdim == 2
  const char* p = reinterpret_cast<const char*>(src + h0 * s.st[2]);
  const int shift = (int)(reinterpret_cast<uintptr_t>(p) & 15);
  const int bytes = n * (int)sizeof(E), head = min(bytes, (16 - shift) & 15), body = (bytes - head) & ~15;
  char* d = dst + shift;
  for (int i = threadIdx.x * 16; i < body; i += SB_NT * 16) small_copy<16>(d + head + i, p + head + i);
  for (int i = threadIdx.x * UNIT; i < head; i += SB_NT * UNIT) small_copy<UNIT>(d + i, p + i);
  for (int i = head + body + threadIdx.x * UNIT; i < bytes; i += SB_NT * UNIT) small_copy<UNIT>(d + i, p + i);
  return shift;
}

template <class R, bool CPLX, int T, bool REG>
__global__ void __launch_bounds__(SB_NT) small_batched_kernel(const __grid_constant__ GemmArgs g,
                                                              const __grid_constant__ SmallArgs p) {
  using E = typename Elem<R, CPLX>::type;
  extern __shared__ __align__(16) unsigned char small_smem[];
  const int64_t h0 = (int64_t)blockIdx.x * p.G;
  const int gcount = (int)(g.H - h0 < p.G ? g.H - h0 : p.G);
  const auto fill = [&](const SmallSide& s, const E* X, char* dst) {
    if (s.linear) return reinterpret_cast<const E*>(dst + small_linear<E, sizeof(R)>(s, X, dst, h0, gcount));
    E* d = reinterpret_cast<E*>(dst);
    if (p.wide)
      small_visit<REG>(s, h0, gcount, [&](int64_t off, int i, int, int, int) { small_copy<sizeof(E)>(d + i, X + off); });
    else
      small_visit<REG>(s, h0, gcount, [&](int64_t off, int i, int, int, int) {
        small_copy<sizeof(R)>(d + i, X + off);
        if (CPLX) small_copy<sizeof(R)>(reinterpret_cast<R*>(d + i) + 1, reinterpret_cast<const R*>(X + off) + 1);
      });
    return reinterpret_cast<const E*>(d);
  };
  const E* sA = fill(p.a, static_cast<const E*>(g.A), reinterpret_cast<char*>(small_smem));
  const E* sB = fill(p.b, static_cast<const E*>(g.B), reinterpret_cast<char*>(small_smem) + p.b_off);
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();

  const int M = (int)g.M, N = (int)g.N, K = (int)g.K;
  const int per = p.mt * p.nt, t = threadIdx.x;
  const int gi = t / per, q = t % per, bm = q % p.mt, bn = q / p.mt;
  const bool mine = gi < gcount;
  R tr[T][T], ti[CPLX ? T : 1][CPLX ? T : 1];
#pragma unroll
  for (int i = 0; i < T; ++i)
#pragma unroll
    for (int j = 0; j < T; ++j) {
      tr[i][j] = R(0);
      if (CPLX) ti[i][j] = R(0);
    }
  if (mine) {
    const E* a[T];
    const E* b[T];
#pragma unroll
    for (int i = 0; i < T; ++i) a[i] = sA + gi * p.as + min(bm + i * p.mt, M - 1) * p.ar;
#pragma unroll
    for (int j = 0; j < T; ++j) b[j] = sB + gi * p.bs + min(bn + j * p.nt, N - 1) * p.bn;
    const R sa = (CPLX && g.conj_a) ? R(-1) : R(1), sb = (CPLX && g.conj_b) ? R(-1) : R(1);
    // FP32 sums restart every 16 k, as in the direct tiles.
    for (int kb = 0; kb < K; kb += 16) {
      R cr[T][T], ci[CPLX ? T : 1][CPLX ? T : 1];
#pragma unroll
      for (int i = 0; i < T; ++i)
#pragma unroll
        for (int j = 0; j < T; ++j) {
          cr[i][j] = sizeof(R) == 4 ? R(0) : tr[i][j];
          if (CPLX) ci[i][j] = sizeof(R) == 4 ? R(0) : ti[i][j];
        }
      const int ke = min(K, kb + 16);
#pragma unroll 2
      for (int k = kb; k < ke; ++k) {
        R ar[T], ai[T], br[T], bi[T];
#pragma unroll
        for (int i = 0; i < T; ++i) {
          Elem<R, CPLX>::load(a[i] + k * p.ak, ar[i], ai[i]);
          ai[i] *= sa;
        }
#pragma unroll
        for (int j = 0; j < T; ++j) {
          Elem<R, CPLX>::load(b[j] + k * p.bk, br[j], bi[j]);
          bi[j] *= sb;
        }
#pragma unroll
        for (int i = 0; i < T; ++i)
#pragma unroll
          for (int j = 0; j < T; ++j) {
            cr[i][j] = fma(ar[i], br[j], cr[i][j]);
            if (CPLX) {
              cr[i][j] = fma(-ai[i], bi[j], cr[i][j]);
              ci[i][j] = fma(ar[i], bi[j], ci[i][j]);
              ci[i][j] = fma(ai[i], br[j], ci[i][j]);
            }
          }
      }
#pragma unroll
      for (int i = 0; i < T; ++i)
#pragma unroll
        for (int j = 0; j < T; ++j) {
          tr[i][j] = sizeof(R) == 4 ? tr[i][j] + cr[i][j] : cr[i][j];
          if (CPLX) ti[i][j] = sizeof(R) == 4 ? ti[i][j] + ci[i][j] : ci[i][j];
        }
    }
  }
  __syncthreads();  // the operands have been read: D takes their place
  E* D = static_cast<E*>(g.D);
  const E* C = static_cast<const E*>(g.C);
  const Epilogue e = g.e;
  // A linear D that is only overwritten leaves as it lies, in 16-byte stores.
  const bool lin = p.d.linear && e.plain;
  char* dp = reinterpret_cast<char*>(D + (lin ? h0 * p.d.st[2] : 0));
  const int shift = lin ? (int)(reinterpret_cast<uintptr_t>(dp) & 15) : 0;
  E* so = reinterpret_cast<E*>(small_smem + shift);
  if (mine) {
#pragma unroll
    for (int i = 0; i < T; ++i)
#pragma unroll
      for (int j = 0; j < T; ++j) {
        const int m = bm + i * p.mt, n = bn + j * p.nt;
        if (m < M && n < N) Elem<R, CPLX>::store(so + gi * p.ds + m * p.dr + n * p.dc, tr[i][j], CPLX ? ti[i][j] : R(0));
      }
  }
  __syncthreads();
  if (lin) {
    const int bytes = gcount * M * N * (int)sizeof(E), head = min(bytes, (16 - shift) & 15), body = (bytes - head) & ~15;
    const char* sp = reinterpret_cast<const char*>(so);
    for (int i = threadIdx.x * 16; i < body; i += SB_NT * 16)
      *reinterpret_cast<uint4*>(dp + head + i) = *reinterpret_cast<const uint4*>(sp + head + i);
    constexpr int U = sizeof(R);
    for (int i = threadIdx.x * U; i < head; i += SB_NT * U)
      *reinterpret_cast<R*>(dp + i) = *reinterpret_cast<const R*>(sp + i);
    for (int i = head + body + threadIdx.x * U; i < bytes; i += SB_NT * U)
      *reinterpret_cast<R*>(dp + i) = *reinterpret_cast<const R*>(sp + i);
    return;
  }
  small_visit<REG>(p.d, h0, gcount, [&](int64_t off, int s, int i0, int i1, int i2) {
    R re, im;
    Elem<R, CPLX>::load(so + s, re, im);
    const E* c = C;
    if (!e.beta_zero) {
      if (REG)
        c += i0 * p.c.st[0] + i1 * p.c.st[1] + i2 * p.c.st[2] + h0 * p.c.st[p.c.hdim];
      else
        c += p.c.vec[0][i0 + (p.c.hdim == 0 ? h0 : 0)] + p.c.vec[1][i1 + (p.c.hdim == 1 ? h0 : 0)] +
             p.c.vec[2][i2 + (p.c.hdim == 2 ? h0 : 0)];
    }
    epilogue_store<R, CPLX>(e, re, im, c, D + off);
  });
}

template <class R, bool CPLX, int T>
cudaError_t run_small(const GemmArgs& g, const SmallArgs& p, bool reg, int bytes, cudaStream_t st) {
  const unsigned grid = (unsigned)((g.H + p.G - 1) / p.G);
  auto kern = reg ? small_batched_kernel<R, CPLX, T, true> : small_batched_kernel<R, CPLX, T, false>;
  if (bytes > 48 * 1024) {
    const cudaError_t r = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (r != cudaSuccess) return r;
  }
  kern<<<grid, SB_NT, bytes, st>>>(g, p);
  return cudaGetLastError();
}

int64_t uabs64(int64_t x) { return x < 0 ? -x : x; }

// The three indexes (batch, r, k) of one side in the order of their strides.
SmallSide small_side(const SmallIndex& h, const SmallIndex& r, const SmallIndex& k, const int* order) {
  const SmallIndex* ix[3] = {&h, &r, &k};
  SmallSide s{};
  for (int i = 0; i < 3; ++i) {
    const int o = order[i];
    s.size[i] = o == 0 ? 0 : (int)ix[o]->n;
    s.st[i] = ix[o]->stride;
    s.vec[i] = ix[o]->vec;
    if (o == 0) s.hdim = i;
  }
  return s;
}
// Whether consecutive batch entries are one contiguous run in this order.
bool small_is_linear(const SmallSide& s) {
  return s.hdim == 2 && (s.size[0] == 1 || s.st[0] == 1) && (s.size[1] == 1 || s.st[1] == s.size[0]) &&
         s.st[2] == (int64_t)s.size[0] * s.size[1];
}
// Shared-memory strides of (batch, r, k) under the order: the memory's own for a
// linear side, else [batch][k][r] with `ld` between depths.
void small_strides(SmallSide& s, const int* order, int linear, int entry, int ld, int* st_h, int* st_r, int* st_k) {
  int* out[3] = {st_h, st_r, st_k};
  const int dense[3] = {entry, 1, ld};
  s.linear = linear;
  int acc = 1;
  for (int i = 0; i < 3; ++i) {
    s.dst[i] = linear ? acc : dense[order[i]];
    *out[order[i]] = s.dst[i];
    if (order[i] != 0) acc *= s.size[i];
  }
}
void small_order(const SmallIndex& h, const SmallIndex& r, const SmallIndex& k, int* order) {
  const SmallIndex* ix[3] = {&h, &r, &k};
  const auto key = [&](int i) { return ix[i]->n < 2 ? INT64_MAX : uabs64(ix[i]->lead); };
  for (int i = 0; i < 3; ++i) order[i] = i;
  for (int i = 0; i < 2; ++i)
    for (int j = 0; j < 2 - i; ++j)
      if (key(order[j + 1]) < key(order[j])) {
        const int x = order[j];
        order[j] = order[j + 1];
        order[j + 1] = x;
      }
}

}  // namespace

cudaError_t launch_small_batched(int dtype, const GemmArgs& g, const SmallLayout& L, cudaStream_t st) {
  if (g.M <= 0 || g.N <= 0 || g.H <= 0) return cudaSuccess;
  if (!small_batched_fits(g.M, g.N, g.K, g.H)) return cudaErrorInvalidValue;
  const int es = dtype == 0 ? 4 : dtype == 3 ? 16 : 8;
  const int M = (int)g.M, N = (int)g.N, K = (int)g.K;
  SmallArgs p{};
  int oa[3], ob[3], od[3];
  small_order(L.h_a, L.a_m, L.a_k, oa);
  small_order(L.h_b, L.b_n, L.b_k, ob);
  small_order(L.h_d, L.d_m, L.d_n, od);
  p.a = small_side(L.h_a, L.a_m, L.a_k, oa);
  p.b = small_side(L.h_b, L.b_n, L.b_k, ob);
  p.d = small_side(L.h_d, L.d_m, L.d_n, od);
  p.c = small_side(L.h_c, L.c_m, L.c_n, od);
  // Odd strides between depths: the element copies of a k-fast operand spread
  // over the banks. A k-fast A' kept linear would put the lanes' rows K
  // elements apart, so it is kept only where K is odd.
  const int ldm = M | 1, ldn = N | 1;
  const bool la = L.regular && small_is_linear(p.a) && (oa[0] == 1 || K % 2 == 1 || M == 1);
  const bool lb = L.regular && small_is_linear(p.b), ld = L.regular && small_is_linear(p.d);
  small_strides(p.a, oa, la, K * ldm, ldm, &p.as, &p.ar, &p.ak);
  small_strides(p.b, ob, lb, K * ldn, ldn, &p.bs, &p.bn, &p.bk);
  small_strides(p.d, od, ld, N * ldm, ldm, &p.ds, &p.dr, &p.dc);
  const int ab = p.as + p.bs, entry = (ab > p.ds ? ab : p.ds) * es;
  // A side with the batch innermost wants whole 32-byte sectors of entries.
  const bool hfast = p.a.hdim == 0 || p.b.hdim == 0 || p.d.hdim == 0;
  int room = SB_SMEM / entry;
  if (hfast && room < 32 / es) room = 96 * 1024 / entry < 32 / es ? 96 * 1024 / entry : 32 / es;
  if (room < 1) room = 1;
  // 4 x 4 outputs a thread where that keeps half the threads of a group busy.
  const int b4 = ((M + 3) / 4) * ((N + 3) / 4), b2 = ((M + 1) / 2) * ((N + 1) / 2);
  const int T = (M * N > 16 && b4 * room >= SB_NT / 2) || b2 > SB_NT ? 4 : 2;
  p.mt = (M + T - 1) / T;
  p.nt = (N + T - 1) / T;
  int G = SB_NT / (p.mt * p.nt);
  if (G > room) G = room;
  if (G > g.H) G = (int)g.H;
  p.G = G;
  p.b_off = (G * p.as * es + 31) & ~15;  // room for the source's offset within 16 bytes
  p.wide = (reinterpret_cast<uintptr_t>(g.A) | reinterpret_cast<uintptr_t>(g.B)) % (uintptr_t)(es) == 0;
  for (SmallSide* s : {&p.a, &p.b, &p.d, &p.c}) s->size[s->hdim] = G;
  const bool reg = L.regular;
  const int bytes = (G * p.ds * es > p.b_off + G * p.bs * es ? G * p.ds * es : p.b_off + G * p.bs * es) + 16;
  switch (dtype * 2 + (T == 4)) {
    case 0: return run_small<float, false, 2>(g, p, reg, bytes, st);
    case 1: return run_small<float, false, 4>(g, p, reg, bytes, st);
    case 2: return run_small<double, false, 2>(g, p, reg, bytes, st);
    case 3: return run_small<double, false, 4>(g, p, reg, bytes, st);
    case 4: return run_small<float, true, 2>(g, p, reg, bytes, st);
    case 5: return run_small<float, true, 4>(g, p, reg, bytes, st);
    case 6: return run_small<double, true, 2>(g, p, reg, bytes, st);
    case 7: return run_small<double, true, 4>(g, p, reg, bytes, st);
  }
  return cudaErrorInvalidValue;
}

}  // namespace dev
}  // namespace tprims
