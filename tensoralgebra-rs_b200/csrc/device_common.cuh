// Small device helpers shared by the kernels: element traits and the
// alpha/beta/conjugation epilogue of one output element.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include "kernels.cuh"

namespace tprims {
namespace dev {

template <class R>
struct Cplx {
  R re, im;
};

// Storage element of a dtype: real R or interleaved complex of R.
template <class R, bool CPLX>
struct Elem;
template <class R>
struct Elem<R, false> {
  using type = R;
  __device__ static inline void load(const type* p, R& re, R& im) {
    re = *p;
    im = R(0);
  }
  __device__ static inline void store(type* p, R re, R) { *p = re; }
};
template <class R>
struct Elem<R, true> {
  using type = Cplx<R>;
  __device__ static inline void load(const type* p, R& re, R& im) {
    re = p->re;
    im = p->im;
  }
  __device__ static inline void store(type* p, R re, R im) {
    type v;
    v.re = re;
    v.im = im;
    *p = v;
  }
};

// One output element: D = op_D(alpha * acc + beta * op_C(C)), with the
// write-back modes of the reference (pack/writeback.rs:311-419): a plain store
// for alpha == 1, beta == 0; alpha scaling only when beta == 0 (C unread); the
// full form otherwise.
template <class R, bool CPLX>
__device__ inline void epilogue_store(const Epilogue& e, R acc_re, R acc_im, const typename Elem<R, CPLX>::type* c,
                                      typename Elem<R, CPLX>::type* d) {
  R vr, vi;
  if (e.plain) {
    vr = acc_re;
    vi = acc_im;
  } else {
    const R ar = (R)e.alpha_re, ai = (R)e.alpha_im;
    if (CPLX) {
      vr = acc_re * ar - acc_im * ai;
      vi = acc_re * ai + acc_im * ar;
    } else {
      vr = acc_re * ar;
      vi = R(0);
    }
    if (!e.beta_zero) {
      R cr, ci;
      Elem<R, CPLX>::load(c, cr, ci);
      if (e.conj_c) ci = -ci;
      const R br = (R)e.beta_re, bi = (R)e.beta_im;
      if (CPLX) {
        vr += cr * br - ci * bi;
        vi += cr * bi + ci * br;
      } else {
        vr += cr * br;
      }
    }
    if (CPLX && e.conj_d) vi = -vi;
  }
  Elem<R, CPLX>::store(d, vr, vi);
}

// ---- f32 as sums of BF16 planes: values that they cannot carry --------------
//
// From the largest (ea, eb) and the smallest non-zero (la, lb; 999: none) exponents
// of a tile's operands: the magnitude below which an output of the split products may
// differ from f32 arithmetic's. 0: none; infinity: every output, for an infinity, a
// NaN, a leading plane that rounds to infinity or a sum of `k` products that could
// overflow. With
// products down to 2^-100 and elements down to 2^-100 every plane and every kept
// product is a normal number; below that, up to 2^-126 times the other operand is
// lost per product, which 2^46 times as much leaves below f32 rounding.
__device__ __forceinline__ float split_guard(int ea, int la, int eb, int lb, int k) {
  // |x| < 2^(ea + 1), so the sum is below 2^(ea + eb + 2 + 32 - clz(k)).
  if (ea >= 127 || eb >= 127 || ea + eb + 34 - __clz(k) > 126) return __uint_as_float(0x7f800000u);
  if (la == 999 || lb == 999 || (la + lb >= -100 && la >= -100 && lb >= -100)) return 0.f;
  const int e = ea > eb ? ea : eb;
  return __uint_as_float((uint32_t)(127 - 80 + (e + 1 > 0 ? e + 1 : 0)) << 23);
}
__device__ __forceinline__ bool split_lost(float thr, float v) {
  return thr != 0.f && !(fabsf(v) >= thr && fabsf(v) < __uint_as_float(0x7f800000u));
}

// Bounded wait on a nanosecond clock (the limit is per wait).
__device__ inline uint64_t globaltimer_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

}  // namespace dev
}  // namespace tprims
