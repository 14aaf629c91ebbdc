// Complex arithmetic, compile-time loops and compile-time twiddle factors
// shared by every kernel of the FAME GB300 library.
//
// Complex values are stored interleaved (re, im) as float2 / double2, the
// layout of MATLAB's interleaved-complex arrays, so one element is one 8- or
// 16-byte vector access.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <cmath>
#include <type_traits>
#include <utility>

#define FAME_HD __host__ __device__ __forceinline__

namespace fame {

// ---------------------------------------------------------------------------
// Double-single ("float-float") real: the unevaluated sum hi + lo of two
// floats, |lo| <= ulp(hi)/2, about 48 significant bits.  Built from the
// error-free transformations of Knuth (two-sum), Dekker (fast two-sum) and
// the FMA two-product (Hida, Li and Bailey's double-double algorithms with
// float in place of double).  On GB300 the FP32 pipes issue 64 times the
// instructions of the FP64 pipe, so an operator evaluated in this type at
// ~20 FP32 instructions per operation is faster than FP64 and as accurate to
// ~1e-14 relative.  (Needs IEEE float arithmetic without reassociation:
// these files are compiled without fast-math.)
// ---------------------------------------------------------------------------
// s + e = a + b exactly (Knuth)
FAME_HD void ff_two_sum(float a, float b, float& s, float& e) {
  s = a + b;
  const float bv = s - a;
  e = (a - (s - bv)) + (b - bv);
}
// s + e = a + b exactly for |a| >= |b| (Dekker)
FAME_HD void ff_fast_two_sum(float a, float b, float& s, float& e) {
  s = a + b;
  e = b - (s - a);
}

// The operators are hidden friends: found for ff operands only, so they never
// take part in float or double expressions.
struct ff {
  float hi, lo;
  FAME_HD constexpr ff() : hi(0.0f), lo(0.0f) {}
  FAME_HD constexpr ff(double d)
      : hi(static_cast<float>(d)), lo(static_cast<float>(d - static_cast<double>(static_cast<float>(d)))) {}
  FAME_HD constexpr ff(float f) : hi(f), lo(0.0f) {}
  FAME_HD constexpr ff(int i) : ff(static_cast<double>(i)) {}
  FAME_HD constexpr ff(float h, float l, bool) : hi(h), lo(l) {}
  FAME_HD explicit operator double() const { return static_cast<double>(hi) + static_cast<double>(lo); }

  friend FAME_HD ff operator+(ff a, ff b) {
    float s1, s2, t1, t2;
    ff_two_sum(a.hi, b.hi, s1, s2);
    ff_two_sum(a.lo, b.lo, t1, t2);
    s2 += t1;
    ff_fast_two_sum(s1, s2, s1, s2);
    s2 += t2;
    ff_fast_two_sum(s1, s2, s1, s2);
    return ff(s1, s2, true);
  }
  friend FAME_HD ff operator-(ff a) { return ff(-a.hi, -a.lo, true); }
  friend FAME_HD ff operator-(ff a, ff b) { return a + (-b); }
  friend FAME_HD ff operator*(ff a, ff b) {
    const float p = a.hi * b.hi;
    float e = fmaf(a.hi, b.hi, -p);  // the exact error of the product
    e = fmaf(a.hi, b.lo, e);
    e = fmaf(a.lo, b.hi, e);
    float s, t;
    ff_fast_two_sum(p, e, s, t);
    return ff(s, t, true);
  }
  // Division and square roots through FP64: only used for per-thread scale
  // factors, never in the per-element arithmetic.
  friend FAME_HD ff operator/(ff a, ff b) { return ff(static_cast<double>(a) / static_cast<double>(b)); }
  friend FAME_HD ff& operator+=(ff& a, ff b) { return a = a + b; }
  friend FAME_HD ff& operator-=(ff& a, ff b) { return a = a - b; }
  friend FAME_HD ff& operator*=(ff& a, ff b) { return a = a * b; }
  friend FAME_HD ff sqrt(ff a) { return ff(::sqrt(static_cast<double>(a))); }
  friend FAME_HD ff rsqrt(ff a) { return ff(1.0 / ::sqrt(static_cast<double>(a))); }
};

// ff(double) and double(ff) by bit operations: the same results, where the
// plain forms take 4 and 3 operations of the FP64 pipe (64 times rarer than FP32
// ones; loading and storing complex128 vectors kept it busy for a third of the
// time of the double-single plane kernels).  Both return false, and leave the
// plain form to the caller, outside the range of exponents that the bits cover.
FAME_HD uint32_t f32_bits(float f) {
  union { float f; uint32_t u; } c;
  c.f = f;
  return c.u;
}
FAME_HD float bits_f32(uint32_t u) {
  union { float f; uint32_t u; } c;
  c.u = u;
  return c.f;
}
// d as its upper and lower 32 bits
FAME_HD bool ff_split_bits(uint32_t dh, uint32_t dl, ff& v) {
  const uint32_t sign = dh & 0x80000000u, mag = dh ^ sign, e = mag >> 20;  // biased exponent
  // hi = d rounded to 24 bits, the remainder r units of 2^(e - 1023 - 52)
  uint32_t h = ((mag - (896u << 20)) << 3) | (dl >> 29);
  uint32_t r = dl & 0x1fffffffu;
  const bool up = r + (h & 1u) > 0x10000000u;  // to nearest, ties to even
  h += up ? 1u : 0u;
  r = up ? 0x20000000u - r : r;
  // r < 2^29 in two exact parts, rounded once
  const float rf = fmaf(bits_f32(0x4b000000u | (r >> 6)) - 8388608.0f, 64.0f,
                        bits_f32(0x4b000000u | (r & 63u)) - 8388608.0f);
  const float unit = bits_f32((((e - (1023 + 52 - 127)) << 23) | sign) ^ (up ? 0x80000000u : 0u));
  const bool zero = (mag | dl) == 0u;
  v.hi = bits_f32(zero ? sign : h | sign);
  v.lo = zero ? 0.0f : rf * unit;
  return zero || (e >= 1023 - 74 && e < 1023 + 127);
}
// f as the upper and lower 32 bits of a double
FAME_HD bool f32_widen_bits(float f, uint32_t& dh, uint32_t& dl) {
  const uint32_t u = f32_bits(f), mag = u & 0x7fffffffu;
  dh = (u & 0x80000000u) | (mag ? (mag >> 3) + (896u << 20) : 0u);
  dl = u << 29;
  return mag == 0u || (mag >= 0x00800000u && mag < 0x7f800000u);
}

struct cff {
  ff x, y;
};

template <class R> struct cx_of;
template <> struct cx_of<float> { using type = float2; };
template <> struct cx_of<double> { using type = double2; };
template <> struct cx_of<ff> { using type = cff; };
template <class R> using cx = typename cx_of<R>::type;

template <class R> FAME_HD cx<R> mk(R a, R b) { cx<R> z; z.x = a; z.y = b; return z; }
template <class R> FAME_HD cx<R> zero() { return mk<R>(R(0), R(0)); }
// a * b + c in one rounding where the type has the instruction (float, double).
FAME_HD float rfma(float a, float b, float c) { return fmaf(a, b, c); }
FAME_HD double rfma(double a, double b, double c) { return fma(a, b, c); }
FAME_HD ff rfma(ff a, ff b, ff c) { return a * b + c; }

// A thread's running sum.  FP32: with the rounding error of every addition kept
// beside it (exactly, Knuth's two-sum), so that a sum of any length carries the
// rounding of its terms and of one final addition; FP64: plain.  The terms are sums over
// a voxel or an element, so a wide batch, whose threads go through many voxels,
// rounds no more than a narrow one.
template <class R> struct RunSum {
  R hi = R(0), lo = R(0);
  FAME_HD void add(R t) {
    const R s = hi + t;
    if constexpr (std::is_same<R, float>::value) {
      const R u = s - hi;
      lo += (hi - (s - u)) + (t - u);
    }
    hi = s;
  }
  // (FP32 on the device: widened by bit operations, one addition of the FP64 pipe; three
  // operations of it per thread and sum cost small solves 1 to 2 %: n = 8, one vector 430 -> 435 us)
  FAME_HD double value() const {
#if defined(__CUDA_ARCH__)
    if constexpr (std::is_same<R, float>::value) {
      uint32_t h[2], l[2];
      if (f32_widen_bits(hi, h[0], l[0]) & f32_widen_bits(lo, h[1], l[1]))
        return __hiloint2double(h[0], l[0]) + __hiloint2double(h[1], l[1]);
    }
#endif
    return double(hi) + double(lo);
  }
};

template <class V> FAME_HD V cadd(V a, V b) { a.x += b.x; a.y += b.y; return a; }
template <class V> FAME_HD V csub(V a, V b) { a.x -= b.x; a.y -= b.y; return a; }
template <class V> FAME_HD V cneg(V a) { a.x = -a.x; a.y = -a.y; return a; }
template <class V> FAME_HD V cconj(V a) { a.y = -a.y; return a; }
template <class V> FAME_HD V cmul(V a, V b) {
  V z; z.x = a.x * b.x - a.y * b.y; z.y = a.x * b.y + a.y * b.x; return z;
}
// conj(a) * b
template <class V> FAME_HD V cmulc(V a, V b) {
  V z; z.x = a.x * b.x + a.y * b.y; z.y = a.x * b.y - a.y * b.x; return z;
}
template <class V, class R> FAME_HD V cscale(V a, R s) { a.x *= s; a.y *= s; return a; }
// a + s*b (real s)
template <class V, class R> FAME_HD V caxpy(R s, V b, V a) {
  a.x = rfma(s, b.x, a.x); a.y = rfma(s, b.y, a.y); return a;
}
// a + i*s*b (real s)
template <class V, class R> FAME_HD V caxpyi(R s, V b, V a) {
  a.x = rfma(-s, b.y, a.x); a.y = rfma(s, b.x, a.y); return a;
}
// a + b*c and a + conj(b)*c: four fused multiply-adds (written out, because
// a + (b.x*c.x - b.y*c.y) contracts to a product, one FMA and an addition:
// six instructions where the FP64 pipe bounds the kernel)
template <class V> FAME_HD V cfma(V b, V c, V a) {
  a.x = rfma(b.x, c.x, rfma(-b.y, c.y, a.x)); a.y = rfma(b.x, c.y, rfma(b.y, c.x, a.y)); return a;
}
template <class V> FAME_HD V cfmac(V b, V c, V a) {
  a.x = rfma(b.x, c.x, rfma(b.y, c.y, a.x)); a.y = rfma(b.x, c.y, rfma(-b.y, c.x, a.y)); return a;
}
FAME_HD cff cfma(cff b, cff c, cff a) {
  a.x += b.x * c.x - b.y * c.y; a.y += b.x * c.y + b.y * c.x; return a;
}
FAME_HD cff cfmac(cff b, cff c, cff a) {
  a.x += b.x * c.x + b.y * c.y; a.y += b.x * c.y - b.y * c.x; return a;
}
// a + i*b (s > 0) or a - i*b (s < 0)
template <int S, class V> FAME_HD V caddi(V a, V b) {
  V z;
  if (S > 0) { z.x = a.x - b.y; z.y = a.y + b.x; } else { z.x = a.x + b.y; z.y = a.y - b.x; }
  return z;
}
// multiply by +i (s>0) or -i (s<0)
template <int S, class V> FAME_HD V cmul_i(V a) {
  V z;
  if (S > 0) { z.x = -a.y; z.y = a.x; } else { z.x = a.y; z.y = -a.x; }
  return z;
}
#if defined(__CUDA_ARCH__) && __CUDA_ARCH__ >= 1000  // host checks compile these headers for other targets
// complex64 on the device: both components in one packed FP32 instruction
// (the FP32 pipe takes the same time for it as for two scalar ones, but it
// costs one issue slot, and the complex64 kernels are bound by issue).
// Forms that swap the components stay scalar: a packed operand would have to
// be assembled by register moves first.
FAME_HD float2 cadd(float2 a, float2 b) { return __fadd2_rn(a, b); }
FAME_HD float2 csub(float2 a, float2 b) { return __ffma2_rn(b, make_float2(-1.0f, -1.0f), a); }
FAME_HD float2 cscale(float2 a, float s) { return __fmul2_rn(a, make_float2(s, s)); }
FAME_HD float2 caxpy(float s, float2 b, float2 a) { return __ffma2_rn(make_float2(s, s), b, a); }
FAME_HD float2 cfma(float2 b, float2 c, float2 a) {
  a = __ffma2_rn(make_float2(b.x, b.x), c, a);
  a.x = fmaf(-b.y, c.y, a.x); a.y = fmaf(b.y, c.x, a.y); return a;
}
FAME_HD float2 cfmac(float2 b, float2 c, float2 a) {
  a = __ffma2_rn(make_float2(b.x, b.x), c, a);
  a.x = fmaf(b.y, c.y, a.x); a.y = fmaf(-b.y, c.x, a.y); return a;
}
FAME_HD float2 cmul(float2 a, float2 b) {
  float2 z = __fmul2_rn(make_float2(a.x, a.x), b);
  z.x = fmaf(-a.y, b.y, z.x); z.y = fmaf(a.y, b.x, z.y); return z;
}
FAME_HD float2 cmulc(float2 a, float2 b) {
  float2 z = __fmul2_rn(make_float2(a.x, a.x), b);
  z.x = fmaf(a.y, b.y, z.x); z.y = fmaf(-a.y, b.x, z.y); return z;
}
#endif
template <class V> FAME_HD double cabs2d(V a) { return double(a.x) * a.x + double(a.y) * a.y; }

template <class D, class S> FAME_HD cx<D> cvt(S a) { return mk<D>(D(a.x), D(a.y)); }

// ---------------------------------------------------------------------------
// Compile-time loop: f(std::integral_constant<int, I>) for I in [B, E).
// ---------------------------------------------------------------------------
template <int B, int E, class F> FAME_HD void static_for(F&& f) {
  if constexpr (B < E) {
    f(std::integral_constant<int, B>{});
    static_for<B + 1, E>(f);
  }
}

// ---------------------------------------------------------------------------
// Compile-time cos / sin of 2*pi*m/n.
//
// Exact integer reduction to the nearest quarter turn, then Taylor series of
// sin and cos on |x| <= pi/4 (terms through x^29, far below one ulp of a
// double).  Evaluated by the compiler only: every call site binds the result
// to a constexpr variable.
// ---------------------------------------------------------------------------
constexpr double kPi = 3.141592653589793238462643383279502884;

// sqrt of a positive integer, by Newton's iteration (compile time)
FAME_HD constexpr double csqrt_int(int n) {
  double r = double(n);
  for (int k = 0; k < 64; ++k) r = 0.5 * (r + double(n) / r);
  return r;
}
FAME_HD constexpr double taylor_sin(double x) {
  double x2 = x * x, term = x, sum = x;
  for (int k = 1; k < 16; ++k) {
    term *= -x2 / double((2 * k) * (2 * k + 1));
    sum += term;
  }
  return sum;
}
FAME_HD constexpr double taylor_cos(double x) {
  double x2 = x * x, term = 1.0, sum = 1.0;
  for (int k = 1; k < 16; ++k) {
    term *= -x2 / double((2 * k - 1) * (2 * k));
    sum += term;
  }
  return sum;
}
// returns cos (which == 0) or sin (which == 1) of 2*pi*m/n
FAME_HD constexpr double cs2pi(long long m, long long n, int which) {
  m %= n;
  if (m < 0) m += n;
  // 4m/n = q + r/n with |r| <= n/2
  long long four_m = 4 * m;
  long long q = (four_m + n / 2) / n;
  long long r = four_m - q * n;
  double th = (kPi / 2.0) * double(r) / double(n);
  double c = taylor_cos(th), s = taylor_sin(th);
  int quad = int(q % 4);
  double cc = quad == 0 ? c : quad == 1 ? -s : quad == 2 ? -c : s;
  double ss = quad == 0 ? s : quad == 1 ? c : quad == 2 ? -s : -c;
  return which == 0 ? cc : ss;
}

}  // namespace fame
