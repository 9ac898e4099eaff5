// fused.cuh -- what the fused transfer-matrix kernels share: their arguments
// and the pointwise factors k(p) and w(x).
#pragma once

#include "common.cuh"
#include "fft.cuh"

namespace nrcps {

struct FusedArgs {
  void* psi;              // [orbitals][V] complex R
  long n_orb_total;       // nconf * batch
  int batch;              // orbitals per configuration
  const float2* kin_f;    // k(p) split as (hi, lo) floats, hi + lo = k to ~1e-15 (R = float)
  const double* kin_d;    // k(p) in FP64 (R = double)
  const double* pos;      // optional P(x)
  const void* zpos;       // Z2 fields with P(x): per site the weights (1 + a) P(x)/V and (1 - a) P(x)/V,
                          // split (hi, lo, hi, lo) as float4 for R = float, (plus, minus) double2 for double
  int field_mode;         // 1 bits, 2 complex phi, 0 complex fld, 3 real FP32 weights (FP32 orbitals)
  const void* field;
  uint64_t off0;          // element/bit offset of configuration 0
  uint64_t conf_stride;
  const uint64_t* conf_base;  // optional per-configuration offsets (replace conf * conf_stride)
  double a;
  double vol;
  double inv_vol;          // 1 / vol (a product per site instead of a division)
  double w_plus, w_minus;  // (1 + a)/V and (1 - a)/V for Z2 fields
  int* err;                // device flag: 1 = a bounded wait timed out
  unsigned long long wait_ns;  // time limit of every mbarrier wait (%globaltimer nanoseconds)
  int stall_test;          // 1: the first wait of CTA 0 of cluster 0 is on an mbarrier nothing arrives on
};

// x * (wr + i wi)
template <typename R>
__device__ __forceinline__ cplx<R> mul_w(cplx<R> x, double wr, double wi) {
  R rh, rl, ih, il;
  split<R>(wr, rh, rl);
  if (wi == 0.0) return scale2<R>(x, rh, rl);  // real weight (Z2, Gaussian, potential): the same value, half the work
  split<R>(wi, ih, il);
  // (x.re + i x.im)(wr + i wi) with each real product taken correctly rounded
  cplx<R> y;
  y.re = mul2<R>(x.re, rh, rl) - mul2<R>(x.im, ih, il);
  y.im = mul2<R>(x.re, ih, il) + mul2<R>(x.im, rh, rl);
  return y;
}

// x * w for the position-space factor of site `site` (general modes).
template <typename R>
__device__ __forceinline__ cplx<R> apply_w_general(const FusedArgs& f, uint64_t kb, int site, cplx<R> x) {
  double wr, wi;
  const uint64_t k = kb + (uint64_t)site;
  if (sizeof(R) == 4 && f.field_mode == 3) {  // the site's weight, made once per run
    const float w = __ldg(reinterpret_cast<const float*>(f.field) + k);
    // rounded products (never fused into a following add): every kind gives
    // the same values
    return cplx<R>{(R)__fmul_rn((float)x.re, w), (R)__fmul_rn((float)x.im, w)};
  }
  if (f.field_mode == 1) {
    uint32_t word = __ldg(reinterpret_cast<const uint32_t*>(f.field) + (k >> 5));
    wr = ((word >> (k & 31)) & 1u) ? f.w_plus : f.w_minus;
    wi = 0.0;
  } else if (f.field_mode == 2) {
    double2 phi = __ldg(reinterpret_cast<const double2*>(f.field) + k);
    wr = (1.0 + f.a * phi.x) * f.inv_vol;
    wi = (f.a * phi.y) * f.inv_vol;
  } else {
    double2 v = __ldg(reinterpret_cast<const double2*>(f.field) + k);
    wr = v.x;
    wi = v.y;
  }
  if (f.pos) {
    double p = __ldg(f.pos + site);
    wr *= p;
    wi *= p;
  }
  return mul_w<R>(x, wr, wi);
}

// x * w(x) along a pencil of L sites STRIDE apart from `site0`: the values of
// apply_w_general.  Complex fields are loaded eight sites (four beside FP64
// pencils at L = 24, for want of registers) ahead of their use and asked together whether their weights
// are real: apply_w_general's branch holds each load back until the site
// before is done, L trips to L2 one after the other.  FP32, L = 32, 3800
// orbitals, Gaussian field: 931 us a step against 1624 (chunks of 16: 1065); FP64,
// L = 24, 627: 150 against 168 (of two: 153); L = 48, 510: 943 against 1179 (of
// four: 1005).  A weight table (mode 3) has its own loop for the same reason:
// through apply_w_general's branches an FP32 batch of 42 configurations of 33
// orbitals at L = 24 took 31.1 ms, now 23.4.
template <typename R, int L, int STRIDE>
__device__ __forceinline__ void apply_w_pencil(const FusedArgs& f, uint64_t kb, int site0, cplx<R>* x) {
  constexpr int CH = sizeof(R) == 8 && L == 24 ? 4 : 8;
  static_assert(L % CH == 0, "whole chunks");
  if constexpr (sizeof(R) == 4) {
    if (f.field_mode == 3) {  // (rounded products, as apply_w_general's)
      const float* tab = reinterpret_cast<const float*>(f.field) + kb + (uint64_t)site0;
#pragma unroll
      for (int i = 0; i < L; ++i) {
        const float w = __ldg(tab + i * STRIDE);
        x[i] = cplx<R>{(R)__fmul_rn((float)x[i].re, w), (R)__fmul_rn((float)x[i].im, w)};
      }
      return;
    }
  }
  if (f.field_mode == 1) {
#pragma unroll
    for (int i = 0; i < L; ++i) x[i] = apply_w_general<R>(f, kb, site0 + i * STRIDE, x[i]);
    return;
  }
  const double2* field = reinterpret_cast<const double2*>(f.field) + kb + (uint64_t)site0;
  const bool phi = f.field_mode == 2;
#pragma unroll
  for (int c = 0; c < L; c += CH) {
    double2 v[CH];
#pragma unroll
    for (int i = 0; i < CH; ++i) v[i] = __ldg(field + (c + i) * STRIDE);
    bool real = true;
#pragma unroll
    for (int i = 0; i < CH; ++i) {
      if (phi) {
        v[i].x = (1.0 + f.a * v[i].x) * f.inv_vol;
        v[i].y = (f.a * v[i].y) * f.inv_vol;
      }
      if (f.pos) {
        const double p = __ldg(f.pos + site0 + (c + i) * STRIDE);
        v[i].x *= p;
        v[i].y *= p;
      }
      real = real && v[i].y == 0.0;
    }
    if (real) {  // (mul_w's product for a real weight)
#pragma unroll
      for (int i = 0; i < CH; ++i) {
        R hi, lo;
        split<R>(v[i].x, hi, lo);
        x[c + i] = scale2<R>(x[c + i], hi, lo);
      }
    } else {
#pragma unroll
      for (int i = 0; i < CH; ++i) x[c + i] = mul_w<R>(x[c + i], v[i].x, v[i].y);
    }
  }
}

template <typename R, bool PK = false>
__device__ __forceinline__ cplx<R> apply_kin(const FusedArgs& f, int site, cplx<R> x) {
  if constexpr (sizeof(R) == 4) {
    float2 k = __ldg(f.kin_f + site);
    if constexpr (PK) return fft::scale2_packed(x, k.x, k.y);
    else return scale2<R>(x, k.x, k.y);
  } else {
    R k = __ldg(f.kin_d + site);
    return cplx<R>{x.re * k, x.im * k};
  }
}

// x * (hi + lo), packed when PK (FP32 only)
template <typename R, bool PK>
__device__ __forceinline__ cplx<R> scale_w(cplx<R> x, R hi, R lo);

// x * w for a Z2 site with a position factor, from the table of both weights
// of every site: the value apply_w_general gives (the table holds the same
// products w_plus * P and w_minus * P, split the same way)
template <typename R>
struct ZposEntry {
  typedef double2 type;
};
template <>
struct ZposEntry<float> {
  typedef float4 type;
};
template <typename R, bool PK>
__device__ __forceinline__ cplx<R> scale_w_entry(typename ZposEntry<R>::type t, bool up, cplx<R> x) {
  if constexpr (sizeof(R) == 4) return scale_w<R, PK>(x, up ? t.x : t.z, up ? t.y : t.w);
  else return scale_w<R, PK>(x, up ? t.x : t.y, (R)0);
}
template <typename R, bool PK>
__device__ __forceinline__ cplx<R> scale_w_zpos(const void* tab, int site, bool up, cplx<R> x) {
  return scale_w_entry<R, PK>(__ldg(reinterpret_cast<const typename ZposEntry<R>::type*>(tab) + site), up, x);
}

// x * (hi + lo), packed when PK (FP32 only)
template <typename R, bool PK>
__device__ __forceinline__ cplx<R> scale_w(cplx<R> x, R hi, R lo) {
  if constexpr (PK && sizeof(R) == 4) return fft::scale2_packed(x, hi, lo);
  else return scale2<R>(x, hi, lo);
}

// x * w for a weight that one float holds exactly (lo = 0): the same value
// as scale_w(x, w, 0), in one product per component.  The products are
// rounded, never fused into a following add: every scalar kind gives the same
// values, whatever its transform does next.
template <typename R, bool PK>
__device__ __forceinline__ cplx<R> scale_w1(cplx<R> x, R w) {
  if constexpr (PK && sizeof(R) == 4) {
    const float2 r = __fmul2_rn(make_float2(x.re, x.im), make_float2(w, w));
    return cplx<R>{r.x, r.y};
  } else {
    if constexpr (sizeof(R) == 4) return cplx<R>{(R)__fmul_rn((float)x.re, (float)w), (R)__fmul_rn((float)x.im, (float)w)};
    else return cplx<R>{__dmul_rn(x.re, w), __dmul_rn(x.im, w)};
  }
}

// Prefetch of a global range into L2 by the bulk copy engine (no completion).
__device__ __forceinline__ void prefetch_l2(const void* p, uint32_t bytes) {
  asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p), "r"(bytes) : "memory");
}

}  // namespace nrcps
