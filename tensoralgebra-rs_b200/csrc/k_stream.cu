// Gather-fed stream tiles: the direct (no pack pass) plain kernels for single
// launches with many tiles of short or moderate K, and for grouped lists.
//
// A tile of such a contraction is a few dozen K steps, so a kernel that runs
// scatter loads, gathers, products and write-back one after another in every
// CTA leaves the arithmetic pipe idle for most of a tile. Here a CTA is
// persistent and warp-specialised: one producer warp walks the CTA's tiles and
// gathers their operand stages through the scatter vectors with cp.async into
// a ring of shared-memory stages, running ahead across tile boundaries; the
// compute warps only wait for full stages, multiply and write back, so the next
// tile's index loads and gathers overlap this tile's products and epilogue.
//
//   producer: tile -> row offsets in registers; per stage 16 k offsets in one
//             register per lane (fetched a stage ahead, passed by shuffles);
//             an operand's copies of 16 bytes where its elements lie side by
//             side along rows or k, else one cp.async per element, into [k][row]
//             order; the tile's output offsets go to a double-buffered slot by
//             cp.async with the first stage.
//   compute:  full[stage] -> fragments -> empty[stage]; after the last stage
//             the epilogue from the slot, then slot_empty.
//
// Only the k of the last stage that exist are multiplied (in steps of four), so a
// short odd K costs no padded depth. Every mbarrier wait is bounded by %globaltimer
// (a status bit, then the role ends); the producer drains its own copies before it
// exits.
#include "tc_common.cuh"

namespace tprims {
namespace dev {

namespace {

using namespace tc;

__device__ __forceinline__ void cpa8(uint32_t dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cpa8z(uint32_t dst, const void* src, bool ok) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(dst), "l"(src), "r"(ok ? 8 : 0) : "memory");
}
// 16-byte copy of `bytes` (0, a multiple of the element, or 16), the rest zero-filled.
__device__ __forceinline__ void cpa16z(uint32_t dst, const void* src, int bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
// The barrier's pending count drops by one when this thread's earlier cp.async
// copies have landed.
__device__ __forceinline__ void cpa_arrive(uint64_t* bar) {
  asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void cpa_drain() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// Shared-memory order of an operand's stage (16 deep):
//   rows-fast operands: [k][row], row stride LD elements;
//   k-fast operands: 128-byte rows of 16 k, the 16-byte chunk c of row
//   r at chunk c xor (r mod 8) (the order TMA's SWIZZLE_128B gives the packed
//   panels): a copy of 16 consecutive k of a row is one contiguous write, and the
//   fragment reads (8 rows x 4 k) are free of bank conflicts.
//
// One operand's gather of a stage: ROWS x 16 elements of ES bytes. A warp copy
// covers 32 rows of one k (rows fast) or 16 consecutive k of two rows (k fast),
// so it touches two or three 128-byte lines; with `vec` (the host found every
// offset a multiple of 16 bytes and the fast index contiguous) the copies are
// 16 bytes wide and half as many. The row offsets of the tile stay
// in registers, one row per lane, and reach the lanes by shuffles, as the
// stage's k offsets do. Rows past the operand's end are left as they are (their
// products are never stored); k past the range are zero-filled.
template <int ES, int ROWS, int LD>
struct StageGather {
  static constexpr int RREG = (ROWS + 31) / 32, V = 16 / ES;
  int64_t off[RREG];  // row lane + 32 j

  __device__ __forceinline__ void init(const int64_t* rows, int64_t r0, int64_t nrows, int lane) {
    const int64_t last = nrows - 1 - r0;
#pragma unroll
    for (int j = 0; j < RREG; ++j) {
      const int64_t r = lane + 32 * j;
      off[j] = __ldg(rows + r0 + (r < last ? r : last)) * ES;
    }
  }
  // kreg: lanes 0..15 (and 16..31 again) hold the stage's k offsets in bytes;
  // kv: k of the stage that exist; rv: rows of the tile that exist.
  __device__ __forceinline__ void issue(const char* base, uint32_t dst, int64_t kreg, int kv, int rv, int kfast,
                                        int vec, int lane) const {
    if (kfast) {
      if (vec) {
        const int c = lane & 7, rl = lane >> 3;  // chunk of two k, row of four
        const int64_t ko = __shfl_sync(0xffffffffu, kreg, 2 * c);
        const char* p = base + ko;
        const int sz = min(max(kv - 2 * c, 0), 2) * 8;
#pragma unroll
        for (int j = 0; j < ROWS / 4; ++j) {
          const int64_t ro = __shfl_sync(0xffffffffu, off[RREG > 1 ? j / 8 : 0], (4 * j + rl) & 31);
          const int row = 4 * j + rl;
          if (row < rv) cpa16z(dst + (uint32_t)(row * 128 + ((c ^ (row & 7)) << 4)), p + ro, sz);
        }
      } else {
        const int kk = lane & 15, rl = lane >> 4;
        const char* p = base + kreg;
        const bool ok = kk < kv;
#pragma unroll
        for (int j = 0; j < ROWS / 2; ++j) {
          const int64_t ro = __shfl_sync(0xffffffffu, off[RREG > 1 ? j / 16 : 0], (2 * j + rl) & 31);
          const int row = 2 * j + rl;
          if (row < rv)
            cpa8z(dst + (uint32_t)(row * 128 + ((((kk >> 1) ^ (row & 7)) << 4) | ((kk & 1) << 3))), p + ro, ok);
        }
      }
      return;
    }
    if (vec) {
      // V rows per copy: lanes cover VL copies of a row range, 32 / VL k at once.
      constexpr int VL = ROWS / V <= 8 ? 8 : ROWS / V <= 16 ? 16 : 32, KP = 32 / VL, NV = (ROWS / V + VL - 1) / VL;
      static_assert(ROWS % V == 0, "whole groups");
      const int r = (lane % VL) * V;
#pragma unroll
      for (int q = 0; q < NV; ++q) {
        const int row = r + q * VL * V;
        int64_t ro = 0;
#pragma unroll
        for (int j = 0; j < RREG; ++j) {
          const int64_t x = __shfl_sync(0xffffffffu, off[j], row & 31);
          if (row / 32 == j) ro = x;
        }
        const int sz = min(max(min(rv, ROWS) - row, 0), V) * ES;
        const char* p = base + ro;
        const uint32_t d = dst + (uint32_t)((lane / VL) * LD + row) * ES;
#pragma unroll
        for (int k0 = 0; k0 < 16; k0 += KP) {
          const int kk = k0 + lane / VL;
          const int64_t ko = __shfl_sync(0xffffffffu, kreg, kk);
          if (sz > 0) cpa16z(d + (uint32_t)(k0 * LD) * ES, p + ko, kk < kv ? sz : 0);
        }
      }
    } else {
#pragma unroll
      for (int kk = 0; kk < 16; ++kk) {
        const int64_t ko = __shfl_sync(0xffffffffu, kreg, kk);
        const bool ok = kk < kv;
        const char* p = base + ko;
        const uint32_t d = dst + (uint32_t)(kk * LD + lane) * ES;
#pragma unroll
        for (int j = 0; j < RREG; ++j)
          if (lane + 32 * j < rv) cpa8z(d + 32 * j * ES, p + off[j], ok);
      }
    }
  }
};

__device__ __forceinline__ void dmma_k8(double (&d)[4], const double (&a)[4], const double (&b)[2]) {
  asm volatile("mma.sync.aligned.m16n8k8.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
               "{%0,%1,%2,%3};\n"
               : "+d"(d[0]), "+d"(d[1]), "+d"(d[2]), "+d"(d[3])
               : "d"(a[0]), "d"(a[1]), "d"(a[2]), "d"(a[3]), "d"(b[0]), "d"(b[1]));
}
__device__ __forceinline__ void dmma_k4(double (&d)[4], double a0, double a1, double b) {
  asm volatile("mma.sync.aligned.m16n8k4.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%0,%1,%2,%3};\n"
               : "+d"(d[0]), "+d"(d[1]), "+d"(d[2]), "+d"(d[3])
               : "d"(a0), "d"(a1), "d"(b));
}

// Output offsets of one tile (double-buffered): written by the producer with
// the tile's first stage, read by the epilogue.
template <int BM, int BN>
struct __align__(16) TileSlot {
  int64_t dm[BM], cm[BM], dn[BN], cn[BN];
  int64_t h, m0, n0, split;
  int nk;      // stages; 0 ends the CTA
  int kv;      // k of the last stage
  int item;    // of a grouped list

};

// f64 on the DMMA pipe: WGM x WGN warps of TI x TJ m16n8 tiles.
template <int WGM, int WGN, int TI, int TJ, int STG, int MINB_>
struct StreamF64 {
  using R = double;
  static constexpr int ES = 8, WARPS = WGM * WGN, BM = WGM * TI * 16, BN = WGN * TJ * 8, BK = 16;
  // Row strides of 4 (mod 16) doubles: the fragment reads (8 rows x 4 k) are
  // free of bank conflicts.
  static constexpr int SA = BM + 4, SB = BN % 16 == 0 ? BN + 4 : BN + 12;
  static constexpr int STAGES = STG, MINB = MINB_;
  static constexpr int A_BYTES = BK * SA * 8, B_BYTES = BK * SB * 8;

  double acc[TI][TJ][4];
  int wm0, wn0, fr, fk;

  __device__ __forceinline__ StreamF64(int warp, int lane)
      : wm0((warp % WGM) * TI * 16), wn0((warp / WGM) * TJ * 8), fr(lane >> 2), fk(lane & 3) {}
  __device__ __forceinline__ void clear() {
#pragma unroll
    for (int i = 0; i < TI; ++i)
#pragma unroll
      for (int j = 0; j < TJ; ++j)
#pragma unroll
        for (int q = 0; q < 4; ++q) acc[i][j][q] = 0.0;
  }
  // Fragment addresses under either stage order: k part (four values per
  // thread) plus a row step per eight rows.
  struct Side {
    int k[2][2], step;  // [ks][r]: k = 8 ks + 4 r + fk; elements
  };
  __device__ __forceinline__ void side(Side& d, int swz, int ld, int w0) const {
    d.step = swz ? 8 * 16 : 8;
#pragma unroll
    for (int ks = 0; ks < 2; ++ks)
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        const int k = 8 * ks + 4 * r + fk;
        d.k[ks][r] = swz ? (w0 + fr) * 16 + ((((k >> 1) ^ fr) << 1) | (k & 1)) : k * ld + w0 + fr;
      }
  }
  Side da, db;
  __device__ __forceinline__ void tile_begin(const GemmArgs& g) {
    side(da, g.a_kfast, SA, wm0);
    side(db, g.b_kfast, SB, wn0);
  }
  __device__ __forceinline__ void k8(const double* A, const double* B, int ks) {
    double a[TI][4], b[TJ][2];
#pragma unroll
    for (int i = 0; i < TI; ++i)
#pragma unroll
      for (int r = 0; r < 4; ++r) a[i][r] = A[da.k[ks][r >> 1] + da.step * (2 * i + (r & 1))];
#pragma unroll
    for (int j = 0; j < TJ; ++j)
#pragma unroll
      for (int r = 0; r < 2; ++r) b[j][r] = B[db.k[ks][r] + db.step * j];
#pragma unroll
    for (int i = 0; i < TI; ++i)
#pragma unroll
      for (int j = 0; j < TJ; ++j) dmma_k8(acc[i][j], a[i], b[j]);
  }
  // The first four k of the half `ks`.
  __device__ __forceinline__ void k4(const double* A, const double* B, int ks) {
#pragma unroll
    for (int j = 0; j < TJ; ++j) {
      const double b = B[db.k[ks][0] + db.step * j];
#pragma unroll
      for (int i = 0; i < TI; ++i)
        dmma_k4(acc[i][j], A[da.k[ks][0] + da.step * (2 * i)], A[da.k[ks][0] + da.step * (2 * i + 1)], b);
    }
  }
  __device__ __forceinline__ void stage(const char* sA, const char* sB, int kv) {
    const double* A = reinterpret_cast<const double*>(sA);
    const double* B = reinterpret_cast<const double*>(sB);
    if (kv > 4)
      k8(A, B, 0);
    else
      k4(A, B, 0);
    if (kv > 12)
      k8(A, B, 1);
    else if (kv > 8)
      k4(A, B, 1);
  }
  __device__ __forceinline__ void store(const GemmArgs& g, const TileSlot<BM, BN>& s) {
    const int mrem = (int)min((int64_t)BM, g.M - s.m0), nrem = (int)min((int64_t)BN, g.N - s.n0);
    if (g.partial) {
      double* P = static_cast<double*>(g.partial) + ((s.split * g.H + s.h) * g.N + s.n0) * g.M + s.m0;
      each([&](int rr, int cc, double v) {
        if (rr < mrem && cc < nrem) P[cc * g.M + rr] = v;
      });
      return;
    }
    double* Db = static_cast<double*>(g.D) + g.s.h_d[s.h];
    if (g.e.plain) {
      // The overwrite form, kept small: the general form below is several
      // times its code, and a tile's epilogue runs once per few stages.
#pragma unroll
      for (int j = 0; j < TJ; ++j) {
        const int cc = wn0 + j * 8 + fk * 2;
        double* d0 = Db + s.dn[cc];
        double* d1 = Db + s.dn[cc + 1];
#pragma unroll
        for (int i = 0; i < TI; ++i)
#pragma unroll
          for (int q = 0; q < 2; ++q) {
            const int rr = wm0 + i * 16 + fr + 8 * q;
            const int64_t dm = s.dm[rr];
            if (rr < mrem && cc < nrem) d0[dm] = acc[i][j][2 * q];
            if (rr < mrem && cc + 1 < nrem) d1[dm] = acc[i][j][2 * q + 1];
          }
      }
      return;
    }
    const double* Cb = static_cast<const double*>(g.C) + (g.e.beta_zero ? 0 : g.s.h_c[s.h]);
    const Epilogue e = g.e;
    each([&](int rr, int cc, double v) {
      if (rr < mrem && cc < nrem)
        epilogue_store<double, false>(e, v, 0.0, Cb + s.cm[rr] + s.cn[cc], Db + s.dm[rr] + s.dn[cc]);
    });
  }
  template <class F>
  __device__ __forceinline__ void each(F&& f) const {
#pragma unroll
    for (int i = 0; i < TI; ++i)
#pragma unroll
      for (int j = 0; j < TJ; ++j)
#pragma unroll
        for (int q = 0; q < 4; ++q) f(wm0 + i * 16 + fr + 8 * (q >> 1), wn0 + j * 8 + fk * 2 + (q & 1), acc[i][j][q]);
  }
};

template <class Op>
struct StreamSmem {
  static constexpr int STAGE = Op::A_BYTES + Op::B_BYTES;
  static constexpr int SLOT = (int)sizeof(TileSlot<Op::BM, Op::BN>);
  static constexpr int BARS = 2 * Op::STAGES + 4;
  static constexpr int BYTES = Op::STAGES * STAGE + 2 * SLOT + 2 * (int)sizeof(GemmArgs) + BARS * 8 + 16;
  static_assert(STAGE % 16 == 0 && SLOT % 16 == 0, "aligned parts");
};

// GROUPED: tiles are claimed from `counter` over the items of a list (the
// producer finds the item of a claimed tile by a 32-way search of
// `tile_start`); otherwise the CTA walks tiles blockIdx.x, + gridDim.x, ... of
// the one contraction in `gp` (column tile fastest, then row tile, batch, K
// split).
template <class Op, bool GROUPED>
__device__ __forceinline__ void stream_tiles(const GemmArgs& gp, const GroupItem* __restrict__ items,
                                             const int64_t* __restrict__ tile_start, int nitems,
                                             unsigned long long* counter, unsigned* status) {
  constexpr int BM = Op::BM, BN = Op::BN, BK = Op::BK, STAGES = Op::STAGES, ES = Op::ES;
  using SM = StreamSmem<Op>;
  using Slot = TileSlot<BM, BN>;
  extern __shared__ __align__(16) unsigned char stream_smem[];
  char* ring = reinterpret_cast<char*>(stream_smem);
  Slot* slots = reinterpret_cast<Slot*>(stream_smem + STAGES * SM::STAGE);
  GemmArgs* slot_g = reinterpret_cast<GemmArgs*>(stream_smem + STAGES * SM::STAGE + 2 * SM::SLOT);
  uint64_t* full = reinterpret_cast<uint64_t*>(stream_smem + STAGES * SM::STAGE + 2 * SM::SLOT + 2 * sizeof(GemmArgs));
  uint64_t* empty = full + STAGES;
  uint64_t* slot_full = empty + STAGES;
  uint64_t* slot_empty = slot_full + 2;

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&full[s], 32);
      mbar_init(&empty[s], Op::WARPS);
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(&slot_full[s], 1);
      mbar_init(&slot_empty[s], Op::WARPS);
    }
    fence_barrier_init();
  }
  __syncthreads();

  if (warp >= Op::WARPS) {
    // ------------------------------------------------------------ producer
    const int64_t total = GROUPED ? tile_start[nitems] : 0;
    const uint64_t t_start = globaltimer_ns();
    constexpr uint64_t LIMIT_NS = 60000000000ull;  // 60 s for one launch
    unsigned long long claim = 0;
    if (GROUPED && lane == 0) claim = atomicAdd(counter, 1ull);
    const int64_t tn1 = (gp.N + BN - 1) / BN, tm1 = (gp.M + BM - 1) / BM;
    const int64_t total1 = tn1 * tm1 * gp.H * (gp.k_chunk ? (gp.K + gp.k_chunk - 1) / gp.k_chunk : 1);
    int stage = 0;
    uint32_t sround = 0;  // completed passes over the ring (its parity gates `empty`)
    for (int64_t it = 0;; ++it) {
      const int sl = (int)(it & 1);
      const uint32_t sl_round = (uint32_t)(it >> 1);
      Slot& slot = slots[sl];
      int64_t h = 0, mt = 0, nt = 0, split = 0;
      int item = 0;
      bool end = false;
      if (GROUPED) {
        const int64_t c = (int64_t)__shfl_sync(0xffffffffu, claim, 0);
        if (c >= total) {
          end = true;
        } else {
          if (lane == 0) claim = atomicAdd(counter, 1ull);
          int lo = 0, hi = nitems - 1;
          while (lo < hi) {
            const int step = (hi - lo + 32) / 32;
            const int pos = lo + lane * step;
            const bool le = pos <= hi && tile_start[pos] <= c;
            const unsigned m = __ballot_sync(0xffffffffu, le) | 1u;
            lo += (31 - __clz(m)) * step;
            hi = min(hi, lo + step - 1);
          }
          const GroupItem& gi = items[lo];
          const int64_t local = c - tile_start[lo], tn = gi.tiles_n, tm = gi.tiles_m;
          if (local < 0 || local >= tn * tm * gi.g.H || it > total) {
            if (lane == 0) atomicOr(status, STATUS_BAD_ARGUMENT);
            end = true;
          } else if (globaltimer_ns() - t_start > LIMIT_NS) {
            if (lane == 0) atomicOr(status, STATUS_WAIT_TIMEOUT);
            end = true;
          }
          end = __any_sync(0xffffffffu, end);
          if (!end) {
            if (local < 0x7fffffff && tm * tn < 0x7fffffff) {
              const uint32_t l = (uint32_t)local, per = (uint32_t)(tm * tn), n32 = (uint32_t)tn;
              const uint32_t hq = l / per, r = l - hq * per, mq = r / n32;
              h = hq;
              mt = mq;
              nt = r - mq * n32;
            } else {
              h = local / (tm * tn);
              mt = (local / tn) % tm;
              nt = local % tn;
            }
            item = lo;
          }
        }
      } else {
        const int64_t t = blockIdx.x + it * gridDim.x;
        if (t >= total1) {
          end = true;
        } else if (total1 < 0x7fffffff) {
          // 32-bit divisions: a 64-bit one is over a hundred instructions of
          // the producer's serial chain.
          const uint32_t r = (uint32_t)t / (uint32_t)tn1, z = r / (uint32_t)tm1;
          nt = (uint32_t)t - r * (uint32_t)tn1;
          mt = r - z * (uint32_t)tm1;
          if (z > 0) {
            split = z / (uint32_t)gp.H;
            h = z - (uint32_t)split * (uint32_t)gp.H;
          }
        } else {
          nt = t % tn1;
          const int64_t r = t / tn1;
          mt = r % tm1;
          const int64_t z = r / tm1;
          h = z % gp.H;
          split = z / gp.H;
        }
      }
      const GemmArgs& g = GROUPED ? items[item].g : gp;
      int64_t kb = 0, kspan = 0, m0 = 0, n0 = 0;
      StageGather<ES, BM, Op::SA> ga;
      StageGather<ES, BN, Op::SB> gb;
      const int klane = lane & 15;
      int64_t ka = 0, kbr = 0, ha = 0, hb = 0;
      if (!end) {
        // The tile's index loads start before the wait for the slot.
        m0 = mt * BM;
        n0 = nt * BN;
        kb = g.k_chunk ? split * g.k_chunk : 0;
        kspan = (g.k_chunk ? min(g.K, kb + g.k_chunk) : g.K) - kb;
        ga.init(g.s.a_m, m0, g.M, lane);
        gb.init(g.s.b_n, n0, g.N, lane);
        const int64_t k0 = kb + (klane < kspan ? klane : 0);
        ka = __ldg(g.s.a_k + k0) * ES;
        kbr = __ldg(g.s.b_k + k0) * ES;
        ha = __ldg(g.s.h_a + h) * ES;
        hb = __ldg(g.s.h_b + h) * ES;
      }
      const int nk = end ? 0 : (int)((kspan + BK - 1) / BK), kvl = (int)(kspan - (int64_t)(nk - 1) * BK);
      // The slot's previous tile has been written back.
      if (!mbar_wait(&slot_empty[sl], (sl_round & 1u) ^ 1u)) {
        atomicOr(status, STATUS_WAIT_TIMEOUT);
        break;
      }
      if (lane == 0) {
        slot.nk = nk;
        slot.kv = kvl;
        slot.h = h;
        slot.m0 = m0;
        slot.n0 = n0;
        slot.split = split;
        slot.item = item;
        mbar_arrive(&slot_full[sl]);
      }
      __syncwarp();
      if (end) break;
      if (GROUPED) {
        // The item's arguments, for the compute warps.
        const uint32_t dst = smem_u32(&slot_g[sl]);
        for (int w = lane; w < (int)(sizeof(GemmArgs) / 8); w += 32)
          cpa8(dst + 8 * w, reinterpret_cast<const char*>(&g) + 8 * w);
      }
      // Output offsets, with the first stage's copies.
      if (!g.partial) {
        const bool cread = !g.e.beta_zero;
#pragma unroll
        for (int j = 0; j < (BM + 31) / 32; ++j) {
          const int64_t m = min(m0 + lane + 32 * j, g.M - 1);
          if (BM % 32 != 0 && lane + 32 * j >= BM) break;
          cpa8(smem_u32(&slot.dm[lane + 32 * j]), g.s.d_m + m);
          if (cread) cpa8(smem_u32(&slot.cm[lane + 32 * j]), g.s.c_m + m);
        }
#pragma unroll
        for (int j = 0; j < (BN + 31) / 32; ++j) {
          const int64_t n = min(n0 + lane + 32 * j, g.N - 1);
          if (BN % 32 != 0 && lane + 32 * j >= BN) break;
          cpa8(smem_u32(&slot.dn[lane + 32 * j]), g.s.d_n + n);
          if (cread) cpa8(smem_u32(&slot.cn[lane + 32 * j]), g.s.c_n + n);
        }
      }
      const int arv = (int)min((int64_t)BM, g.M - m0), brv = (int)min((int64_t)BN, g.N - n0);
      const int a_kfast = g.a_kfast, b_kfast = g.b_kfast, a_vec = g.a_vec, b_vec = g.b_vec;
      const char* Ab = static_cast<const char*>(g.A) + ha;
      const char* Bb = static_cast<const char*>(g.B) + hb;
      const int64_t* ak = g.s.a_k + kb + klane;
      const int64_t* bk = g.s.b_k + kb + klane;
      bool alive = true;
      for (int i = 0; i < nk; ++i) {
        const int64_t kac = ka, kbc = kbr;
        const int64_t kn = (int64_t)(i + 1) * BK;
        if (kn + klane < kspan) {
          ka = __ldg(ak + kn) * ES;
          kbr = __ldg(bk + kn) * ES;
        }
        if (!mbar_wait(&empty[stage], (sround & 1u) ^ 1u)) {
          alive = false;
          break;
        }
        const uint32_t dst = smem_u32(ring + stage * SM::STAGE);
        const int kv = i + 1 < nk ? BK : kvl;
        ga.issue(Ab, dst, kac, kv, arv, a_kfast, a_vec, lane);
        gb.issue(Bb, dst + Op::A_BYTES, kbc, kv, brv, b_kfast, b_vec, lane);
        cpa_arrive(&full[stage]);
        if (++stage == STAGES) {
          stage = 0;
          ++sround;
        }
      }
      if (!__all_sync(0xffffffffu, alive)) {
        atomicOr(status, STATUS_WAIT_TIMEOUT);
        break;
      }
    }
    cpa_drain();  // no copy of this warp is in flight when the CTA ends
  } else {
    // ------------------------------------------------------------- compute
    Op op(warp, lane);
    int stage = 0;
    uint32_t sround = 0;
    for (int64_t it = 0;; ++it) {
      const int sl = (int)(it & 1);
      if (!mbar_wait(&slot_full[sl], (uint32_t)(it >> 1) & 1u)) {
        atomicOr(status, STATUS_WAIT_TIMEOUT);
        break;
      }
      const Slot& slot = slots[sl];
      const int nk = slot.nk;
      if (nk == 0) break;
      const int kvl = slot.kv;
      op.clear();
      op.tile_begin(GROUPED ? items[slot.item].g : gp);
      bool alive = true;
      for (int i = 0; i < nk; ++i) {
        if (!mbar_wait(&full[stage], sround & 1u)) {
          alive = false;
          break;
        }
        const char* sA = ring + stage * SM::STAGE;
        op.stage(sA, sA + Op::A_BYTES, i + 1 < nk ? BK : kvl);
        __syncwarp();
        if (lane == 0) mbar_arrive(&empty[stage]);
        if (++stage == STAGES) {
          stage = 0;
          ++sround;
        }
      }
      if (!__all_sync(0xffffffffu, alive)) {
        atomicOr(status, STATUS_WAIT_TIMEOUT);
        break;
      }
      op.store(GROUPED ? slot_g[sl] : gp, slot);
      __syncwarp();
      if (lane == 0) mbar_arrive(&slot_empty[sl]);
    }
  }
}

// One contraction: parameters within 288 bytes (above, a launch costs the host 0.6 us more;
// f64 547 x 1061 x 2 9.9 -> 8.95 us a call, the direct tile 8.75).
template <class Op>
__global__ void __launch_bounds__(Op::WARPS * 32 + 32, Op::MINB)
stream_kernel(const __grid_constant__ GemmArgs g) {
  stream_tiles<Op, false>(g, nullptr, nullptr, 0, nullptr, g.status);
}

template <class Op>
__global__ void __launch_bounds__(Op::WARPS * 32 + 32, Op::MINB)
stream_group_kernel(const GroupItem* __restrict__ items, const int64_t* __restrict__ tile_start, int nitems,
                    unsigned long long* counter, unsigned* status) {
  const GemmArgs none{};
  stream_tiles<Op, true>(none, items, tile_start, nitems, counter, status);
}

template <class Op>
cudaError_t run_stream(const GemmArgs& g, cudaStream_t st) {
  auto kern = stream_kernel<Op>;
  cudaError_t r = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, StreamSmem<Op>::BYTES);
  if (r != cudaSuccess) return r;
  int dev = 0, sms = 148;
  if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const int64_t splits = g.k_chunk ? (g.K + g.k_chunk - 1) / g.k_chunk : 1;
  const int64_t tiles = ((g.N + Op::BN - 1) / Op::BN) * ((g.M + Op::BM - 1) / Op::BM) * g.H * splits;
  const int64_t resident = (int64_t)sms * Op::MINB;
  const unsigned grid = (unsigned)(tiles < resident ? tiles : resident);
  kern<<<grid, Op::WARPS * 32 + 32, StreamSmem<Op>::BYTES, st>>>(g);
  return cudaGetLastError();
}

// The grouped kernel's image is loaded and its attribute set before any capture.
template <class Op>
cudaError_t prepare_group() {
  return cudaFuncSetAttribute(stream_group_kernel<Op>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              StreamSmem<Op>::BYTES);
}
template <class Op>
cudaError_t run_group(const GroupItem* items, const int64_t* tile_start, int nitems, unsigned long long* counter,
                      unsigned* status, int num_sms, cudaStream_t st) {
  stream_group_kernel<Op><<<num_sms * Op::MINB, Op::WARPS * 32 + 32, StreamSmem<Op>::BYTES, st>>>(
      items, tile_start, nitems, counter, status);
  return cudaGetLastError();
}

using SF64_64x64 = StreamF64<2, 2, 2, 4, 4, 3>;
using SF64_128x32 = StreamF64<4, 1, 2, 4, 3, 3>;
using SF64_64x48 = StreamF64<4, 1, 1, 6, 4, 3>;
using SF64_32x128 = StreamF64<1, 4, 2, 4, 3, 3>;

// The roles of A' and B' (and of the output's rows and columns) exchanged.
GemmArgs swapped(const GemmArgs& g) {
  GemmArgs t = g;
  t.s.a_m = g.s.b_n;
  t.s.a_k = g.s.b_k;
  t.s.b_k = g.s.a_k;
  t.s.b_n = g.s.a_m;
  t.s.c_m = g.s.c_n;
  t.s.c_n = g.s.c_m;
  t.s.d_m = g.s.d_n;
  t.s.d_n = g.s.d_m;
  t.s.h_a = g.s.h_b;
  t.s.h_b = g.s.h_a;
  t.s.blk_a_m = g.s.blk_b_n;
  t.s.blk_a_k = g.s.blk_b_k;
  t.s.blk_b_k = g.s.blk_a_k;
  t.s.blk_b_n = g.s.blk_a_m;
  t.A = g.B;
  t.B = g.A;
  t.M = g.N;
  t.N = g.M;
  t.conj_a = g.conj_b;
  t.conj_b = g.conj_a;
  t.a_kfast = g.b_kfast;
  t.b_kfast = g.a_kfast;
  t.a_vec = g.b_vec;
  t.b_vec = g.a_vec;
  t.a_ld = g.b_ld;
  t.b_ld = g.a_ld;
  t.d_mfast = 1;
  return t;
}

struct StreamFamily {
  int dtype, bm, bn;
  const char* name;
};
const StreamFamily kStream[] = {
    {1, 64, 64, "sm100.f64.dmma884.stream.64x64x16"},   {1, 128, 32, "sm100.f64.dmma884.stream.128x32x16"},
    {1, 64, 48, "sm100.f64.dmma884.stream.64x48x16"},   {1, 32, 128, "sm100.f64.dmma884.stream.32x128x16"},
    {0, 128, 128, "sm100.f32.tcgen05.stream.128x128x32"}, {2, 64, 128, "sm100.c32.tcgen05.stream.64x128x32"},
    {0, 128, 256, "sm100.f32.tcgen05.tma.split.128x256x32"}, {2, 64, 256, "sm100.c32.tcgen05.tma.split.64x256x32"},
};

}  // namespace

bool is_stream_kernel(int kernel) { return kernel >= PLAIN_STREAM_FIRST && kernel <= PLAIN_STREAM_LAST; }
void stream_tile_shape(int kernel, int* bm, int* bn) {
  *bm = kStream[kernel - PLAIN_STREAM_FIRST].bm;
  *bn = kStream[kernel - PLAIN_STREAM_FIRST].bn;
}
int stream_dtype(int kernel) { return kStream[kernel - PLAIN_STREAM_FIRST].dtype; }
const char* stream_kernel_name(int kernel) { return kStream[kernel - PLAIN_STREAM_FIRST].name; }

// Each family's padded outputs, weighted by its measured time per padded
// output relative to 64 x 64 (B200, 177147 x 243 x 50 f64: 64 x 64 0.201
// ms, 128 x 32 0.234, 64 x 48 0.259 on 1.13 times the padded area, 32 x 128 0.208).
int choose_stream_kernel(int dtype, int64_t M, int64_t N, const LaunchHints& hints, double* waste) {
  static const struct {
    int kernel;
    double weight;
  } table[] = {{PLAIN_F64_STREAM_64x64, 1.0},   {PLAIN_F64_STREAM_128x32, 1.15}, {PLAIN_F64_STREAM_64x48, 1.15},
               {PLAIN_F64_STREAM_32x128, 1.03}};
  const int64_t m = hints.d_mfast ? M : N, n = hints.d_mfast ? N : M;  // the launch's roles
  int best = 0;
  for (const auto& f : table) {
    if (stream_dtype(f.kernel) != dtype) continue;
    int bm = 0, bn = 0;
    stream_tile_shape(f.kernel, &bm, &bn);
    const double w = f.weight * (double)((m + bm - 1) / bm * bm) * (double)((n + bn - 1) / bn * bn) / ((double)m * (double)n);
    if (!best || w < *waste) {
      best = f.kernel;
      *waste = w;
    }
  }
  return best;
}

// Rows of the tile run along D's unit-stride index (the lanes' stores).
GemmArgs stream_oriented(const GemmArgs& g) { return !g.d_mfast && !g.partial ? swapped(g) : g; }

cudaError_t prepare_stream_grouped(int kernel) {
  switch (kernel) {
    case PLAIN_F64_STREAM_64x64: return prepare_group<SF64_64x64>();
    case PLAIN_F64_STREAM_128x32: return prepare_group<SF64_128x32>();
    case PLAIN_F64_STREAM_64x48: return prepare_group<SF64_64x48>();
    case PLAIN_F64_STREAM_32x128: return prepare_group<SF64_32x128>();
  }
  return cudaErrorInvalidValue;
}

cudaError_t launch_stream_grouped(int kernel, const GroupItem* items, const int64_t* tile_start, int nitems,
                                  unsigned long long* counter, unsigned* status, int num_sms, cudaStream_t st) {
  switch (kernel) {
    case PLAIN_F64_STREAM_64x64: return run_group<SF64_64x64>(items, tile_start, nitems, counter, status, num_sms, st);
    case PLAIN_F64_STREAM_128x32: return run_group<SF64_128x32>(items, tile_start, nitems, counter, status, num_sms, st);
    case PLAIN_F64_STREAM_64x48: return run_group<SF64_64x48>(items, tile_start, nitems, counter, status, num_sms, st);
    case PLAIN_F64_STREAM_32x128: return run_group<SF64_32x128>(items, tile_start, nitems, counter, status, num_sms, st);
  }
  return cudaErrorInvalidValue;
}

cudaError_t launch_stream_gemm(int dtype, int kernel, const GemmArgs& g0, cudaStream_t st) {
  if (g0.M <= 0 || g0.N <= 0 || g0.H <= 0) return cudaSuccess;
  if (g0.K <= 0 || stream_dtype(kernel) != dtype) return cudaErrorInvalidValue;
  const GemmArgs g = stream_oriented(g0);
  switch (kernel) {
    case PLAIN_F64_STREAM_64x64: return run_stream<SF64_64x64>(g, st);
    case PLAIN_F64_STREAM_128x32: return run_stream<SF64_128x32>(g, st);
    case PLAIN_F64_STREAM_64x48: return run_stream<SF64_64x48>(g, st);
    case PLAIN_F64_STREAM_32x128: return run_stream<SF64_32x128>(g, st);
  }
  return cudaErrorInvalidValue;
}

}  // namespace dev
}  // namespace tprims
