// Compensated FP32 arithmetic for complex128 data ("float-float", error-free
// transformations).
//
// GB300 executes FP64 at 1.2 TFLOP/s but FP32 at 70 TFLOP/s (measured), so a complex128
// gate (16 FP64 FMAs per amplitude) is FP64-bound at 18 % of the HBM roofline. The
// kernels that use this header keep complex128 in HBM, but compute on the FP32 pipe:
//
//   * a double x is split, with integer instructions only, into floats hi + lo where
//     hi is x truncated to 24 significant bits and lo the next 24 bits rounded to
//     nearest, so |x - (hi + lo)| <= 2^-48 |x|;
//   * a product a*b of two split numbers is p + e with p = fl(ah*bh) and
//     e = (ah*bh - p) + ah*bl + al*bh + al*bl, the first term exact by FMA
//     (Dekker's TwoProduct with a fused multiply-add);
//   * sums of the high parts use Knuth's TwoSum (exact: s + err = a + b), the
//     low-order terms are summed in plain FP32;
//   * the result pair is renormalised and turned back into a double with integer
//     instructions plus one FP64 add.
//
// For the magnitudes allowed by in_range() (state elements 0 or 2^-90..2^90, gate
// elements 0 or 2^-30..2^30) every intermediate is a normal float and the relative
// error of a complex multiply-accumulate chain of length 4 is ~2^-46 or better; the
// kernels fall back to native FP64 for a group that has anything outside that range.
// (References: T. J. Dekker, "A floating-point technique for extending the available
// precision", 1971; D. E. Knuth, TAOCP vol. 2, 4.2.2; Ogita, Rump, Oishi, "Accurate
// sum and dot product", 2005.)
#pragma once

#include <stdint.h>
#include <string.h>

#ifdef __CUDACC__
#define DF_HD __host__ __device__ __forceinline__
#else
#define DF_HD inline
#endif

namespace qtnh_impl {
namespace df {

DF_HD uint64_t d2u(double x) {
#ifdef __CUDA_ARCH__
  return (uint64_t)__double_as_longlong(x);
#else
  uint64_t u;
  memcpy(&u, &x, 8);
  return u;
#endif
}
DF_HD double u2d(uint64_t u) {
#ifdef __CUDA_ARCH__
  return __longlong_as_double((long long)u);
#else
  double x;
  memcpy(&x, &u, 8);
  return x;
#endif
}
DF_HD uint32_t f2u(float x) {
#ifdef __CUDA_ARCH__
  return (uint32_t)__float_as_uint(x);
#else
  uint32_t u;
  memcpy(&u, &x, 4);
  return u;
#endif
}
DF_HD float u2f(uint32_t u) {
#ifdef __CUDA_ARCH__
  return __uint_as_float(u);
#else
  float x;
  memcpy(&x, &u, 4);
  return x;
#endif
}

// Correctly rounded single operations that the compiler may not fuse.
DF_HD float add(float a, float b) {
#ifdef __CUDA_ARCH__
  return __fadd_rn(a, b);
#else
  volatile float r = a + b;
  return r;
#endif
}
DF_HD float sub(float a, float b) {
#ifdef __CUDA_ARCH__
  return __fsub_rn(a, b);
#else
  volatile float r = a - b;
  return r;
#endif
}
DF_HD float mul(float a, float b) {
#ifdef __CUDA_ARCH__
  return __fmul_rn(a, b);
#else
  volatile float r = a * b;
  return r;
#endif
}
DF_HD float fma(float a, float b, float c) {
#ifdef __CUDA_ARCH__
  return __fmaf_rn(a, b, c);
#else
  return __builtin_fmaf(a, b, c);
#endif
}

struct f2 {
  float h, l;  // value h + l
};

// A double as its two 32-bit words (hi: sign, 11-bit exponent, top 20 mantissa bits).
// The fast paths test and split doubles through these words only, so no comparison
// or select on a double value reaches the FP64 pipe.
struct dwords {
  uint32_t hi, lo;
};

DF_HD dwords words(double x) {
  uint64_t u = d2u(x);
  return {(uint32_t)(u >> 32), (uint32_t)u};
}

// In range: zero, or biased exponent in [1023 - 90, 1023 + 90] (|x| in [2^-90, 2^91)).
DF_HD bool in_range_state(dwords w) {
  const uint32_t u = w.hi << 1;  // exponent at bits 21-31
  return u - (933u << 21) < (181u << 21) || (u | w.lo) == 0u;
}
// Gate elements: zero or |x| in [2^-30, 2^31).
DF_HD bool in_range_gate(dwords w) {
  const uint32_t u = w.hi << 1;
  return u - (993u << 21) < (61u << 21) || (u | w.lo) == 0u;
}
DF_HD bool in_range_state(double x) { return in_range_state(words(x)); }
DF_HD bool in_range_gate(double x) { return in_range_gate(words(x)); }

DF_HD uint32_t funnel_left3(uint32_t lo, uint32_t hi) {
#ifdef __CUDA_ARCH__
  return __funnelshift_l(lo, hi, 3);
#else
  return (hi << 3) | (lo >> 29);
#endif
}

// x -> hi + lo for an in-range x (see in_range_*). hi is x truncated to 24 significant
// bits: the funnel shift lines up the low 8 exponent bits and 23 mantissa bits, and
// for biased exponents e in [897, 1150] the float exponent e - 896 equals those 8 bits
// with the top bit flipped. lo is the remaining 29 mantissa bits r (weight 2^(E-52),
// E = e - 1023) rounded to 24 bits: r = r1 * 2^6 + r0 is turned into two exact floats
// by the magic-number trick, 2^(E-23) + r1 * 2^(E-46) - 2^(E-23) and
// 2^(E-29) + r0 * 2^(E-52) - 2^(E-29), whose sum is rounded once.
DF_HD f2 split(dwords w) {
  if (((w.hi << 1) | w.lo) == 0u) return {0.0f, 0.0f};
  const uint32_t sgn = w.hi & 0x80000000u;
  const uint32_t f = funnel_left3(w.lo, w.hi);  // low 9 exponent bits at 23-31
  const uint32_t hi = ((f & 0x7FFFFFFFu) | sgn) ^ 0x40000000u;
  const uint32_t c1 = (f & 0xFF800000u) - (919u << 23);  // 2^(E-23): (e - 919) << 23 (mod 2^32)
  const uint32_t c0 = c1 - (6u << 23);            // 2^(E-29)
  const float lo_hi = sub(u2f(c1 | ((w.lo >> 6) & 0x7FFFFFu)), u2f(c1));
  const float lo_lo = sub(u2f(c0 | (w.lo & 63u)), u2f(c0));
  const float lo = add(lo_hi, lo_lo);
  return {u2f(hi), u2f(f2u(lo) | sgn)};
}
DF_HD f2 split(double x) { return split(words(x)); }

// TwoSum (Knuth): s + err == a + b exactly.
DF_HD void two_sum(float a, float b, float& s, float& err) {
  s = add(a, b);
  float bb = sub(s, a);
  err = add(sub(a, sub(s, bb)), sub(b, bb));
}

// Product of two split reals: p + e ~ a*b with p = fl(ah*bh).
DF_HD void two_prod(f2 a, f2 b, float& p, float& e) {
  p = mul(a.h, b.h);
  e = fma(a.h, b.h, -p);
  e = fma(a.h, b.l, e);
  e = fma(a.l, b.h, e);
  e = fma(a.l, b.l, e);
}

// Accumulator for a real sum of products: value s + c.
struct acc {
  float s, c;
};

DF_HD acc acc_first(f2 a, f2 b) {
  acc r;
  two_prod(a, b, r.s, r.c);
  return r;
}

DF_HD void acc_mac(acc& r, f2 a, f2 b) {
  float p, e, s, err;
  two_prod(a, b, p, e);
  two_sum(r.s, p, s, err);
  r.s = s;
  r.c = add(r.c, add(err, e));
}

// 2^-896 times the float u (its exponent bits taken as a double's): exact, zero and
// subnormal floats included.
DF_HD double scaled_double(uint32_t u) {
  const uint32_t hi = (uint32_t)((int32_t)u >> 3) & 0x8FFFFFFFu;
  return u2d(((uint64_t)hi << 32) | (u << 29));
}
// 2^896 d, 0 for a subnormal d (a sum of floats below 2^-126).
DF_HD double unscaled_double(double d) {
  const dwords w = words(d);
  const bool nz = (w.hi & 0x7FF00000u) != 0u;
  const uint32_t hi = nz ? w.hi + (896u << 20) : w.hi & 0x80000000u;
  return u2d(((uint64_t)hi << 32) | (nz ? w.lo : 0u));
}

// s + c rounded once to double: both parts convert exactly, and the one FP64 add
// (two per complex element) uses the FP64 pipe that the rest of the path leaves idle.
DF_HD double to_double(acc r) { return unscaled_double(scaled_double(f2u(r.s)) + scaled_double(f2u(r.c))); }

DF_HD f2 renorm(acc r) {
  f2 v;
  two_sum(r.s, r.c, v.h, v.l);
  return v;
}

// Complex value as four floats.
struct cf2 {
  f2 re, im;
};

DF_HD cf2 csplit(double re, double im) { return {split(re), split(im)}; }

DF_HD f2 neg(f2 a) { return {-a.h, -a.l}; }

// Complex product of split numbers: (a * b) as two accumulators.
DF_HD void cmul_acc(cf2 a, cf2 b, acc& re, acc& im) {
  re = acc_first(a.re, b.re);
  acc_mac(re, a.im, neg(b.im));
  im = acc_first(a.re, b.im);
  acc_mac(im, a.im, b.re);
}

#ifdef __CUDACC__
// ---- two float-float numbers per instruction ---------------------------------------
// Packed FP32 instructions (add/mul/fma.f32x2) do two correctly rounded operations in one
// issue slot. The kernels of this header are bound by instruction issue, so the real and
// imaginary parts of a complex accumulator (or two elements of a stream) go through one
// instruction stream; every result has the bits of the scalar form above.
struct x2 {
  uint64_t v;
};

__device__ __forceinline__ x2 pack(float a, float b) {
  x2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void unpack(x2 p, float& a, float& b) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(p.v));
}
__device__ __forceinline__ x2 add2(x2 a, x2 b) {
  x2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ x2 sub2(x2 a, x2 b) {
  x2 r;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ x2 mul2(x2 a, x2 b) {
  x2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ x2 fma2(x2 a, x2 b, x2 c) {
  x2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
  return r;
}

// Right operand of packed products: high parts, and high and low parts negated (the error
// of a product is formed as p - a b, so that no product has to be negated).
struct rhs2 {
  x2 h, nh, nl;
};
__device__ __forceinline__ rhs2 make_rhs(f2 a, f2 b) { return {pack(a.h, b.h), pack(-a.h, -b.h), pack(-a.l, -b.l)}; }

// Left operand: high and low parts.
struct lhs2 {
  x2 h, l;
};

// Two accumulators: values s - nc.
struct acc2 {
  x2 s, nc;
};

// p = fl(ah bh), ne = p - a b (two_prod with the error negated).
__device__ __forceinline__ void two_prod2(lhs2 a, const rhs2& b, x2& p, x2& ne) {
  p = mul2(a.h, b.h);
  ne = fma2(a.h, b.nh, p);
  ne = fma2(a.h, b.nl, ne);
  ne = fma2(a.l, b.nh, ne);
  ne = fma2(a.l, b.nl, ne);
}
__device__ __forceinline__ acc2 acc2_first(lhs2 a, const rhs2& b) {
  acc2 r;
  two_prod2(a, b, r.s, r.nc);
  return r;
}
__device__ __forceinline__ void acc2_mac(acc2& r, lhs2 a, const rhs2& b) {
  x2 p, ne;
  two_prod2(a, b, p, ne);
  const x2 s = add2(r.s, p), bb = sub2(s, r.s);
  const x2 err = add2(sub2(r.s, sub2(s, bb)), sub2(p, bb));
  r.s = s;
  r.nc = add2(r.nc, sub2(ne, err));
}
// The two sums, each rounded once to double (to_double).
__device__ __forceinline__ void to_double2(const acc2& r, double& a, double& b) {
  float sa, sb, ca, cb;
  unpack(r.s, sa, sb);
  unpack(r.nc, ca, cb);
  a = unscaled_double(scaled_double(f2u(sa)) - scaled_double(f2u(ca)));
  b = unscaled_double(scaled_double(f2u(sb)) - scaled_double(f2u(cb)));
}

__device__ __forceinline__ x2 neg2(x2 a) { return {a.v ^ 0x8000000080000000ull}; }
__device__ __forceinline__ rhs2 make_rhs(x2 h, x2 l) { return {h, neg2(h), neg2(l)}; }

// Two complex products a b (cmul_acc), `a` as its real and imaginary parts, b's parts (and the
// negated imaginary ones) as right operands.
__device__ __forceinline__ void cmul2(lhs2 ar, lhs2 ai, const rhs2& br, const rhs2& bi, const rhs2& nbi, acc2& re,
                                      acc2& im) {
  re = acc2_first(ar, br);
  acc2_mac(re, ai, nbi);
  im = acc2_first(ar, bi);
  acc2_mac(im, ai, br);
}
__device__ __forceinline__ lhs2 make_lhs(f2 a, f2 b) { return {pack(a.h, b.h), pack(a.l, b.l)}; }
__device__ __forceinline__ void cmul2(const cf2 (&a)[2], const cf2 (&b)[2], acc2& re, acc2& im) {
  const rhs2 br = make_rhs(b[0].re, b[1].re), bi = make_rhs(b[0].im, b[1].im);
  const rhs2 nbi{bi.nh, bi.h, pack(b[0].im.l, b[1].im.l)};
  cmul2(make_lhs(a[0].re, a[1].re), make_lhs(a[0].im, a[1].im), br, bi, nbi, re, im);
}

// A complex matrix element as left operands of the products with (re, im) and with
// (im, re): (gr, gr) and (-gi, gi).
struct gate2 {
  lhs2 r, i;
};
__device__ __forceinline__ gate2 make_gate2(cf2 g) {
  return {{pack(g.re.h, g.re.h), pack(g.re.l, g.re.l)}, {pack(-g.im.h, g.im.h), pack(-g.im.l, g.im.l)}};
}
// (re, im) += g x, in the order of the scalar kernels: gr x, then gi (i x).
__device__ __forceinline__ void gate2_mac(acc2& r, bool first, const gate2& g, const rhs2& x, const rhs2& ix) {
  if (first) r = acc2_first(g.r, x);
  else acc2_mac(r, g.r, x);
  acc2_mac(r, g.i, ix);
}
#endif

}  // namespace df
}  // namespace qtnh_impl
