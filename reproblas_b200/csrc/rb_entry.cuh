// rb_entry.cuh -- one output entry of the binned gemv / gemm kernels of every element type:
// operand values, the products an entry deposits, the records of partial states and the
// epilogue that combines an entry's products with beta*y (or the caller's binned state).
#pragma once
#include "rb_binned.cuh"
#include "rb_kernels.cuh"

namespace rb {
namespace xb {

template <typename E, bool CX> struct Val { E r, i; };

// Element `idx` of a real or complex (interleaved pair) array; PAIR: as one load, p being aligned to
// pairs.
template <typename E, bool CX, bool PAIR = false>
__device__ __forceinline__ Val<E, CX> ldv(const E* p, long long idx) {
  Val<E, CX> v;
  if constexpr (CX && PAIR && sizeof(E) == 8) {
    const double2 t = __ldg((const double2*)p + idx);
    v.r = t.x;
    v.i = t.y;
  } else if constexpr (CX && PAIR) {
    const float2 t = __ldg((const float2*)p + idx);
    v.r = t.x;
    v.i = t.y;
  } else if constexpr (CX) {
    v.r = __ldg(p + 2 * idx);
    v.i = __ldg(p + 2 * idx + 1);
  } else {
    v.r = __ldg(p + idx);
    v.i = E(0);
  }
  return v;
}

// fl(v * alpha) as the reference forms it.
template <typename E, bool CX>
__device__ __forceinline__ Val<E, CX> scale(Val<E, CX> v, E ar, E ai) {
  using B = BT<E>;
  Val<E, CX> o;
  if constexpr (CX) {
    o.r = B::sub(B::mul(v.r, ar), B::mul(v.i, ai));
    o.i = B::add(B::mul(v.r, ai), B::mul(v.i, ar));
  } else {
    o.r = B::mul(v.r, ar);
    o.i = E(0);
  }
  return o;
}

// The values one product a*b deposits: D = 1 (real) or 2 per component, at column q*D of
// v[component].
template <typename E, bool CX, int KD>
__device__ __forceinline__ void products(Val<E, CX> a, Val<E, CX> b, E (&v)[CX ? 2 : 1][KD],
                                         int q) {
  using B = BT<E>;
  if constexpr (CX) {
    v[0][2 * q] = B::mul(a.r, b.r);
    v[0][2 * q + 1] = B::mul(-a.i, b.i);
    v[1][2 * q] = B::mul(a.r, b.i);
    v[1][2 * q + 1] = B::mul(a.i, b.r);
  } else {
    v[0][q] = B::mul(a.r, b.r);
  }
}

// binned -> value conversion of one component (ddmconv / ssmconv).
template <typename E, int F>
__device__ __forceinline__ E convx(const E* p, const E* c, int inc) {
  if constexpr (sizeof(E) == 8) return conv<F>(p, c, inc);
  else return sconv<F>(p, c, inc);
}

// Finish one output entry from the renormalised state of its products, a[0..NC-1]:
// kOutValue deposits beta*y into it (nothing when beta == 0, y itself when beta == 1;
// rzgemv.c:47-59 starts from binned(beta*y) -- the same multiset, so the same state) and
// writes the converted value to yout; yin holds y (read by the caller, possibly early).
// kOutBinned merges into the caller's state (reference layout: NC-interleaved primaries,
// then carries).
template <typename E, bool CX, int F>
__device__ __forceinline__ void finish_from(Acc<E, F>* a, int mode, const E* yin, E* yout, E br,
                                            E bi, E* yb) {
  constexpr int NC = CX ? 2 : 1;
  using B = BT<E>;
  if (mode == kOutValue) {
    const bool bzero = br == E(0) && (!CX || bi == E(0));
    const bool bone = br == E(1) && (!CX || bi == E(0));
    E init[NC];
    if constexpr (CX) {
      const E yr = yin[0], yi = yin[1];
      if (bone) {
        init[0] = yr;
        init[1] = yi;
      } else {
        init[0] = B::sub(B::mul(yr, br), B::mul(yi, bi));
        init[1] = B::add(B::mul(yr, bi), B::mul(yi, br));
      }
    } else {
      init[0] = bone ? yin[0] : B::mul(yin[0], br);
    }
#pragma unroll
    for (int c = 0; c < NC; c++) {
      if (!bzero) {
        E v[1] = {init[c]};
        a[c].template tile<1>(v, 1);
      }
      a[c].renorm();
      E p[F], q[F];
      a[c].store(p, q, 1);
      yout[c] = convx<E, F>(p, q, 1);
    }
  } else {
#pragma unroll
    for (int c = 0; c < NC; c++) {
      Acc<E, F> prev;
      prev.load(yb + c, yb + NC * F + c, NC);
      prev.merge(a[c]);
      prev.renorm();
      prev.store(yb + c, yb + NC * F + c, NC);
    }
  }
}

template <typename E, bool CX, int F>
__device__ __forceinline__ void finish(Acc<E, F>* a, int mode, E* yv, E br, E bi, E* yb) {
  constexpr int NC = CX ? 2 : 1;
  E yin[NC];
#pragma unroll
  for (int c = 0; c < NC; c++) yin[c] = E(0);
  if (mode == kOutValue && !(br == E(0) && (!CX || bi == E(0)))) {   // beta 0 reads nothing
#pragma unroll
    for (int c = 0; c < NC; c++) yin[c] = yv[c];
  }
  finish_from<E, CX, F>(a, mode, yin, yv, br, bi, yb);
}

template <typename E>
__device__ __forceinline__ E flags_to(unsigned f) {
  if constexpr (sizeof(E) == 8) return __longlong_as_double((long long)f);
  else return __uint_as_float(f);
}
template <typename E>
__device__ __forceinline__ unsigned flags_from(E v) {
  if constexpr (sizeof(E) == 8) return (unsigned)__double_as_longlong(v);
  else return __float_as_uint(v);
}

// Record of one accumulator: F primaries, F carries, the flags word; element q of the record
// at rec[q * stride].
template <typename E, int F>
__device__ __forceinline__ void put_rec(const Acc<E, F>& a, E* rec, long long stride) {
#pragma unroll
  for (int i = 0; i < F; i++) {
    rec[i * stride] = a.pri[i];
    rec[(F + i) * stride] = a.car[i];
  }
  rec[2 * F * stride] = flags_to<E>(a.flags);
}
// Read a record another CTA wrote (through L2).
template <typename E, int F>
__device__ __forceinline__ void read_rec(Acc<E, F>& o, const E* rec, long long stride) {
  o.zero();
#pragma unroll
  for (int i = 0; i < F; i++) {
    o.pri[i] = __ldcg(rec + i * stride);
    o.car[i] = __ldcg(rec + (F + i) * stride);
  }
  o.flags = flags_from<E>(__ldcg(rec + 2 * F * stride));
  o.set_idx_from_pri();
}

}  // namespace xb
}  // namespace rb
