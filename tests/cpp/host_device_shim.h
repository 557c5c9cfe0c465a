// Lets the device math headers compile as host C++ for the CPU checks: CUDA's qualifiers and the few intrinsics
// those headers use.
#pragma once
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>

#define __device__
#define __host__
#define __forceinline__ inline
#define __restrict__
#include <cstdlib>

static inline long long
__double_as_longlong(double x)
{
  long long r;
  std::memcpy(&r, &x, 8);
  return r;
}
static inline double
__longlong_as_double(long long x)
{
  double r;
  std::memcpy(&r, &x, 8);
  return r;
}
static inline int
__float_as_int(float x)
{
  int r;
  std::memcpy(&r, &x, 4);
  return r;
}
static inline unsigned
__float_as_uint(float x)
{
  return (unsigned)__float_as_int(x);
}
static inline float
__uint_as_float(unsigned x)
{
  float r;
  std::memcpy(&r, &x, 4);
  return r;
}
static inline float
__int_as_float(int x)
{
  return __uint_as_float((unsigned)x);
}
static inline float
__fmul_rn(float x, float y)
{
  return x * y;
}
static inline float
__fadd_rn(float x, float y)
{
  return x + y;
}
static inline float
__fmaf_rn(float x, float y, float z)
{
  return fmaf(x, y, z);
}
static inline int
__double2hiint(double x)
{
  return (int)(__double_as_longlong(x) >> 32);
}
static inline int
__double2loint(double x)
{
  return (int)(uint32_t)__double_as_longlong(x);
}
static inline double
__hiloint2double(int hi, int lo)
{
  return __longlong_as_double((long long)(((uint64_t)(uint32_t)hi << 32) | (uint32_t)lo));
}
static inline unsigned
__funnelshift_l(unsigned lo, unsigned hi, unsigned s)
{
  return (unsigned)(((((uint64_t)hi << 32) | lo) << (s & 31)) >> 32);
}
static inline unsigned
__umulhi(unsigned a, unsigned b)
{
  return (unsigned)(((uint64_t)a * b) >> 32);
}
static inline float
rsqrtf(float x)
{
  return 1.0f / sqrtf(x);
}
// the GPU's reciprocal approximations are off by up to this many units in the last place
#ifndef HOST_SEED_UNITS
#define HOST_SEED_UNITS 0
#endif
static int      host_seed_units = HOST_SEED_UNITS;
static unsigned host_seed_count = 0;
static inline float
host_seed(float x)
{
  if (!host_seed_units || !(fabsf(x) > 1.2e-38f && fabsf(x) < 3e38f))
    return x;
  const int k = (int)(++host_seed_count % (unsigned)(2 * host_seed_units + 1)) - host_seed_units;
  return __uint_as_float(__float_as_uint(x) + (unsigned)k);
}
