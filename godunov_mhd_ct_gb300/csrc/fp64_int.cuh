// FP64 operations of the exact path on the integer pipe.
//
// GB300 issues two FP64 lanes per SM and clock against 128 integer lanes, and an IEEE division or square root is
// a sequence of eight or more FP64 instructions, a comparison, minimum or scaling by 2 one each. The functions
// here give the same IEEE results (round to nearest even; checked bit for bit against the CPU's own FP64 unit in
// tests/cpp/fp64_int_check.cpp) from 32-bit integer multiplies, shifts and compares plus one FP32 approximation
// per reciprocal or square root, which leaves the FP64 pipe to the additions and multiplications. Operands outside the range
// that the integer forms cover (subnormal, infinite, NaN, or a result close to over- or underflow) go to the FP64
// instruction through a function that is not inlined: inlined, the compiler would run both and select.
//
// Division: an integer Newton iteration on the divisor's significand (the reciprocal to 60 bits from a 22-bit
// seed), the quotient's 53 bits from a 64-bit product, and the exact remainder to settle the rounding. Square
// root: the same with the reciprocal square root.
#pragma once

#include <cstdint>

namespace gmhd
{

// The long sequences are functions, not inlined: some ninety sites of them made the step's code exceed the
// instruction cache (3D blast 128^3: 35.5 ms a step inlined, 18.7 ms as calls; Orszag-Tang 18.1 and 17.6).
#ifdef __CUDACC__
#define GMHD_CALL static __device__ __noinline__
static inline float
host_seed(float x)
{
  return x;
}
#else
#define GMHD_CALL inline
#endif

GMHD_CALL double
slow_div(double x, double y)
{
  return x / y;
}
GMHD_CALL double
slow_sqrt(double x)
{
  return sqrt(x);
}
GMHD_CALL double
slow_mul(double x, double y)
{
  return x * y;
}
GMHD_CALL double
slow_max(double x, double y)
{
  return fmax(x, y);
}
GMHD_CALL double
slow_min(double x, double y)
{
  return fmin(x, y);
}

// 1 / x and 1 / sqrt(x) of x in [1, 4), results in (0.5, 1]: within 1 and 2 units in the last place as CUDA documents
// them (in the CPU checks host_seed() adds such an error)
__device__ __forceinline__ float
seed_rcp(float x)
{
#ifdef __CUDA_ARCH__
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
#else
  return host_seed(1.0f / x);
#endif
}
__device__ __forceinline__ float
seed_rsqrt(float x)
{
#ifdef __CUDA_ARCH__
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
#else
  return host_seed(1.0f / sqrtf(x));
#endif
}

// high 64 bits of a * b, at most 3 below
__device__ __forceinline__ uint64_t
mulhi_below(uint64_t a, uint64_t b)
{
  const uint32_t ah = (uint32_t)(a >> 32), al = (uint32_t)a, bh = (uint32_t)(b >> 32), bl = (uint32_t)b;
  return (uint64_t)ah * bh + (((uint64_t)ah * bl) >> 32) + (((uint64_t)al * bh) >> 32);
}

__device__ __forceinline__ uint64_t
make64(uint32_t hi, uint32_t lo)
{
  return ((uint64_t)hi << 32) | lo;
}

// A divisor with the reciprocal of its significand: R = 2^127 / (Y 2^11), Y the 53-bit significand, at most 16 below
struct Rcp64
{
  double   y;
  uint64_t R;
};

GMHD_CALL Rcp64
rcp64(double y)
{
  const uint32_t hi = (uint32_t)__double2hiint(y), lo = (uint32_t)__double2loint(y);
  const uint32_t yh = __funnelshift_l(lo, (hi & 0xfffffu) | 0x100000u, 11), yl = lo << 11; // Y << 11
  // seed: the FP32 reciprocal of the leading 24 bits, taken 4 units low so that it is below the true value
  // (the seed is within 1 unit, the truncation of Y adds less than 2)
  const uint32_t rb = __float_as_uint(seed_rcp(__uint_as_float(0x3f800000u | ((yh >> 8) & 0x7fffffu))));
  const uint32_t v = 0x80000000u + ((rb - 0x3f000004u) << 8);
  // two Newton steps, both from below: relative error 2^-20 -> 2^-40 -> 2^-60
  const uint64_t e1 = 0x8000000000000000ull - ((uint64_t)yh * v + __umulhi(yl, v));
  const uint64_t r1 = make64(v, 0u) + (((uint64_t)v * (uint32_t)(e1 >> 12)) >> 19);
  const uint64_t e2 = 0x8000000000000000ull - mulhi_below(make64(yh, yl), r1) - 4u;
  Rcp64          r;
  r.y = y;
  r.R = r1 + (((uint64_t)(uint32_t)(r1 >> 32) * (uint32_t)e2) >> 31);
  return r;
}

// x / d.y
GMHD_CALL double
div64v(double x, Rcp64 d)
{
  const uint32_t hx = (uint32_t)__double2hiint(x), lx = (uint32_t)__double2loint(x);
  const uint32_t hy = (uint32_t)__double2hiint(d.y), ly = (uint32_t)__double2loint(d.y);
  const uint32_t ex = (hx >> 20) & 0x7ffu, ey = (hy >> 20) & 0x7ffu;
  const uint32_t sign = (hx ^ hy) & 0x80000000u;
  const uint32_t e = ex - ey + 1023u;
  if (ex - 1u >= 2046u || ey - 1u >= 2046u || e - 2u >= 2044u)
  {
    if ((hx << 1 | lx) == 0u && ey - 1u < 2046u)
      return __hiloint2double((int)sign, 0);
    return slow_div(x, d.y);
  }
  const uint32_t Xh = (hx & 0xfffffu) | 0x100000u, Yh = (hy & 0xfffffu) | 0x100000u;
  const uint64_t X = make64(Xh, lx), Y = make64(Yh, ly);
  const uint32_t s = X < Y ? 1u : 0u;
  // quotient in [2^63, 2^64), at most 20 below (so rounding it can only come out low)
  const uint64_t t = mulhi_below(make64(__funnelshift_l(lx, Xh, 11), lx << 11), d.R) << s;
  uint64_t       m = (t >> 11) + ((t >> 10) & 1u);
  // remainder X 2^(52 + s) - m Y modulo 2^64; no quotient lies halfway between two doubles
  const int64_t rem = (int64_t)(make64(lx << (20u + s), 0u) - m * Y);
  m += 2 * rem > (int64_t)Y ? 1u : 0u;
  const uint64_t bits = m + make64((e - s - 1u) << 20, 0u);
  return __hiloint2double((int)((uint32_t)(bits >> 32) | sign), (int)(uint32_t)bits);
}

__device__ __forceinline__ double
div64(double x, const Rcp64 & d)
{
  return div64v(x, d);
}
__device__ __forceinline__ double
div64(double x, double y)
{
  return div64(x, rcp64(y));
}

GMHD_CALL double
sqrt64(double a)
{
  const uint32_t hi = (uint32_t)__double2hiint(a), lo = (uint32_t)__double2loint(a);
  if (hi - 0x00100000u >= 0x7fe00000u)
  {
    if ((hi << 1 | lo) == 0u)
      return a;
    return slow_sqrt(a); // negative, subnormal, infinite or NaN
  }
  // a = A / 2^62 * 4^k, A / 2^62 in [1, 4)
  const uint32_t odd = ((hi >> 20) & 1u) ^ 1u;
  const uint32_t mh = (hi & 0xfffffu) | 0x100000u;
  const uint64_t A = make64(mh, lo) << (10u + odd);
  const uint32_t fb = 0x3f800000u + (odd << 23) + (__funnelshift_l(lo, hi & 0xfffffu, 3));
  const uint32_t rb = __float_as_uint(seed_rsqrt(__uint_as_float(fb)));
  const uint32_t y = 0x80000000u + ((rb - 0x3f000006u) << 8); // 1 / sqrt, below the true value
  const uint64_t e1 = 0x4000000000000000ull - mulhi_below((uint64_t)y * y, A);
  const uint64_t y1 = make64(y, 0u) + (((uint64_t)y * (uint32_t)(e1 >> 12)) >> 19);
  const uint64_t s0 = mulhi_below(A, y1);
  const uint32_t d = (uint32_t)((A >> 2) - mulhi_below(s0, s0)) - 4u;
  const uint64_t s1 = s0 + (((uint64_t)d * (uint32_t)(y1 >> 32)) >> 31);
  uint64_t       m = (s1 >> 10) + ((s1 >> 9) & 1u);
  // remainder A 2^42 - m^2 modulo 2^64: above m means sqrt > m + 1/2
  const int64_t rem = (int64_t)((A << 42) - m * m);
  m += rem > (int64_t)m ? 1u : 0u;
  const uint64_t bits = m + make64(((((hi >> 20) + 1023u - odd) >> 1) - 1u) << 20, 0u);
  return __longlong_as_double((long long)bits);
}

// x > 0
__device__ __forceinline__ bool
dpos(double x)
{
  return (uint64_t)__double_as_longlong(x) - 1u < 0x7ff0000000000000ull;
}

// total order of the non-NaN doubles as signed integers (-0 below +0)
__device__ __forceinline__ int64_t
dkey(double x)
{
  const int64_t b = (int64_t)__double_as_longlong(x);
  return b ^ (int64_t)((uint64_t)(b >> 63) >> 1);
}
// exponent field all ones (infinite or NaN)
__device__ __forceinline__ bool
dspecial(double x)
{
  return ((uint32_t)__double2hiint(x) & 0x7ff00000u) == 0x7ff00000u;
}
__device__ __forceinline__ double
dmax(double a, double b)
{
  if (dspecial(a) || dspecial(b))
    return slow_max(a, b);
  return dkey(a) >= dkey(b) ? a : b;
}
__device__ __forceinline__ double
dmin(double a, double b)
{
  if (dspecial(a) || dspecial(b))
    return slow_min(a, b);
  return dkey(a) <= dkey(b) ? a : b;
}
// a > b: NaN compares false; +0 and -0 are equal
__device__ __forceinline__ bool
dgt(double a, double b)
{
  const bool nan = ((uint64_t)__double_as_longlong(a) << 1) > 0xffe0000000000000ull ||
                   ((uint64_t)__double_as_longlong(b) << 1) > 0xffe0000000000000ull;
  const bool zeros = (((uint64_t)__double_as_longlong(a) | (uint64_t)__double_as_longlong(b)) << 1) == 0u;
  return !nan && !zeros && dkey(a) > dkey(b);
}

// x 2^-n, n = 1, 2 or 3
__device__ __forceinline__ double
dscale_down(double x, uint32_t n)
{
  const uint32_t hi = (uint32_t)__double2hiint(x), e = (hi >> 20) & 0x7ffu;
  if (e - (n + 1u) < 2046u - n)
    return __hiloint2double((int)(hi - (n << 20)), __double2loint(x));
  if ((hi << 1 | (uint32_t)__double2loint(x)) == 0u)
    return x;
  return slow_mul(x, n == 1u ? 0.5 : (n == 2u ? 0.25 : 0.125));
}

} // namespace gmhd
