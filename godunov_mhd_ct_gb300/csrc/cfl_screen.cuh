// CFL reduction in FP64 with an FP32 screen, shared by gmhd_inv_dt and gmhd_inv_dt_noalloc.
//
// The reduction wants one FP64 value: the largest cell_inv_dt_fp64 of a block list. GB300 issues two FP64
// lanes per SM and clock, and the formula's divisions and square roots are sequences of them, so evaluating
// it for every cell is bound by the FP64 pipe (256^3: 6.95 ms against 0.16 ms for reading U and B). Here each
// cell first gets FP32 bounds lo <= value <= hi, and the FP64 formula runs only where hi reaches the largest
// known lo: the same maximum, bit for bit (256^3: 0.29 ms a call; 0.40 with rounding conversions to FP32, three square roots
// an axis and the indices divided out for each cell: 597 instructions a cell then, 415 now, two thirds of the issue slots
// taken, HBM at half its rate). Where all cells are within the
// bounds of one another (a uniform state) every cell is still evaluated in FP64, as before.
#pragma once

#include "mhd_math.cuh"

namespace gmhd
{

struct CflBounds
{
  float lo, hi;
};

// FP32 reciprocal square root of a normal x within 2 ulp
__device__ __forceinline__ float
frsqrt_approx(float x)
{
#ifdef __CUDA_ARCH__
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
#else
  return host_seed(1.0f / sqrtf(x));
#endif
}

// x cut to FP32 (relative error below 2^-23), zero below 2^-126; right for |x| < 2^127, which the caller checks: `top`
// collects the largest high word
__device__ __forceinline__ float
cut_to_f32(double x, uint32_t & top)
{
  const uint32_t hi = (uint32_t)__double2hiint(x), lo = (uint32_t)__double2loint(x), mag = hi & 0x7fffffffu;
  top = top > mag ? top : mag;
  const uint32_t bits = (__funnelshift_l(lo, hi, 3) & 0x7fffffffu) ^ 0x40000000u;
  return __uint_as_float((mag < 0x38100000u ? 0u : bits) | (hi & 0x80000000u));
}

// Bounds of cell_inv_dt_fp64 from the cell's conservative state u[5] and its six face values (left and
// right along x, y, z; 2D: the cell-centred Bz twice); 1/dx and
// gamma - 1 (gm1) to FP32 accuracy.
//
// Error model, e = 2^-24: every FP32 input and operation is within 2 e (approximate ones 4 e). The thermal
// energy and the squared field come from differences, so their error is absolute: at most 15 e times
// tot = |E| + kinetic + magnetic energy with the face magnitudes in place of their means. The squared fast
// speed d2 + sqrt(disc) changes by at most twice the change of c^2 or b_n^2 / rho. Its slope in b_t^2 / rho is
// 1/2 + d2 / (2 sqrt(disc)), up to 160 at the limit of disc below, but sqrt(disc) is at least c b_t / sqrt(rho) and the
// error of b_t^2 is 2 b_t times that of b_t (2 e of the face magnitudes M), so that it adds 2 e c M / sqrt(rho) at most, less
// than e (c^2 + M^2 / rho). All of it is within delta = (gamma (gamma - 1) + 2) 32 e tot / rho plus the speed's own rounding,
// which the final factors 1 +- 64 e cover. Cells outside the range where this holds (tiny or huge or non-finite values, or a
// discriminant near zero, where the FP64 formula itself may return NaN, which the maximum ignores) give
// lo = 0, hi = infinity: they are always evaluated.
__device__ __forceinline__ CflBounds
cell_inv_dt_bounds(const double * u, const double * f, int dim, float idx, float gamma0, float gm1, float smallr,
                   float smallp, const Sources & src)
{
  const float E24 = 5.9604645e-8f;
  const float inf = __int_as_float(0x7f800000);
  uint32_t    top = 0u;
  const float a0 = cut_to_f32(f[0], top), a1 = cut_to_f32(f[1], top), b0 = cut_to_f32(f[2], top),
              b1 = cut_to_f32(f[3], top), c0 = cut_to_f32(f[4], top), c1 = cut_to_f32(f[5], top);
  const float Ax = 0.5f * (a0 + a1), Ay = 0.5f * (b0 + b1), Az = 0.5f * (c0 + c1);
  const float Mx = 0.5f * (fabsf(a0) + fabsf(a1)), My = 0.5f * (fabsf(b0) + fabsf(b1)), Mz = 0.5f * (fabsf(c0) + fabsf(c1));
  const float rho = cut_to_f32(u[0], top), en = cut_to_f32(u[1], top);
  const float r = fmaxf(rho, smallr);
#ifdef __CUDA_ARCH__
  const float ir = __fdividef(1.0f, r);
#else
  const float ir = host_seed(1.0f / r);
#endif
  const float vx = cut_to_f32(u[2], top) * ir, vy = cut_to_f32(u[3], top) * ir, vz = cut_to_f32(u[4], top) * ir;
  const float ekin = 0.5f * r * (vx * vx + vy * vy + vz * vz);
  const float sx = Ax * Ax, sy = Ay * Ay, sz = Az * Az;
  const float tot = fabsf(en) + ekin + 0.5f * (Mx * Mx + My * My + Mz * Mz);
  const float p = fmaxf(gm1 * (en - 0.5f * (sx + sy + sz) - ekin), r * smallp);
  const float c2 = gamma0 * p * ir;
  const float bb = (sx + sy + sz) * ir;
  const float d2 = 0.5f * (bb + c2);
  const float h = 0.5f * (bb - c2);
  const float delta = (gamma0 * gm1 + 2.0f) * (32.0f * E24) * tot * ir;
  // d2^2 - c2 bn^2 / rho = h^2 + c2 bt^2 / rho, without the cancellation
  const float disc_min = 1e-5f * d2 * d2 + 4.0f * delta * delta;
  bool        ok = top < 0x47e00000u && rho > 1e-20f && r < 1e20f && tot < 1e30f && d2 > 1e-15f && d2 < 1e15f;
  float       lo = 0.0f, hi = 0.0f, lo2 = 0.0f, hi2 = 0.0f;
#pragma unroll
  for (int d = 0; d < 3; ++d)
  {
    if (d == 2 && dim != 3)
      continue;
    const float bt = d == 0 ? sy + sz : (d == 1 ? sx + sz : sx + sy);
    const float disc = h * h + c2 * (bt * ir);
    ok = ok && disc > disc_min;
    const float cf2 = d2 + disc * frsqrt_approx(disc);
    const float v = fabsf(d == 0 ? vx : (d == 1 ? vy : vz));
    // sqrt(x - delta) >= sqrt(x) - delta / sqrt(x), sqrt(x + delta) <= sqrt(x) + delta / (2 sqrt(x))
    const float rs = frsqrt_approx(cf2), cf = cf2 * rs;
    const float l = fmaxf(cf - delta * rs, 0.0f) + v, g = cf + 0.5f * delta * rs + v;
    lo += l;
    hi += g;
    if (src.gravity)
    {
      lo2 += l * l;
      hi2 += g * g;
    }
  }
  ok = ok && lo > 1e-12f && hi < 1e18f;
  if (src.gravity)
  {
    // factor (sqrt(1 + 2k) + 1) / 2 grows with k = sum|g| dx / sum v_d^2 (floored)
    float gs = fabsf((float)src.g[0]) + fabsf((float)src.g[1]);
    if (dim == 3)
      gs += fabsf((float)src.g[2]);
    const float gd = gs / idx;
    lo *= 0.5f * (sqrtf(1.0f + 2.0f * fmaxf(gd / hi2 * (1.0f - 64.0f * E24), 1e-4f)) + 1.0f);
    hi *= 0.5f * (sqrtf(1.0f + 2.0f * fmaxf(gd / lo2 * (1.0f + 64.0f * E24), 1e-4f)) + 1.0f);
  }
  lo *= idx;
  hi *= idx;
  if (src.viscosity)
  {
    const float v = 4.0f * ((float)src.mu / rho) * idx * idx;
    lo = fmaxf(lo, v);
    hi = fmaxf(hi, v);
  }
  lo *= 1.0f - 64.0f * E24;
  hi *= 1.0f + 64.0f * E24;
  ok = ok && lo < 1e30f && hi < 1e30f;
  return ok ? CflBounds{lo, hi} : CflBounds{0.0f, inf};
}

#ifdef __CUDACC__
// Cells per thread of a screening CTA (256 threads): their upper bounds stay in registers between the screen
// and the FP64 evaluations.
constexpr int kScreenCells = 4;

// Largest cell_inv_dt_fp64 over cells [c0, c0 + 256 kScreenCells) of one block that may exceed the value
// already in *slot (FP64 bits, 0 at first), max-reduced over the CTA into *slot. 256 threads; `dx` is
// evaluated by dx_of() only where a cell is evaluated in FP64 (an FP64 division costs more than the screen).
template <class DxOf>
__device__ __forceinline__ void
screened_inv_dt(const double * __restrict__ Ub, const double * __restrict__ Bb, int dim, int bx, int by, int64_t c0,
                int64_t ncell, int64_t nfx, int64_t nfy, float idx, double gamma0, float gm1, double smallr,
                double smallp, const Sources & src, DxOf dx_of, unsigned long long * slot)
{
  __shared__ float  s_lo[8];
  __shared__ double s_m[8];
  const float       g_f = (float)gamma0, r_f = (float)smallr, p_f = (float)smallp;
  const int         tid = threadIdx.x;
  float             hi[kScreenCells], lo = 0.0f;
  auto              locate = [&](int64_t c, int & i, int & j, int & k) {
    // 32-bit indices: a block's cells fit (checked by the launchers)
    const unsigned cu = (unsigned)c, row = cu / (unsigned)bx;
    i = (int)(cu - row * (unsigned)bx);
    k = (int)(row / (unsigned)by);
    j = (int)(row - (unsigned)k * (unsigned)by);
  };
  // the cell 256 further on: no division but for the first
  const unsigned left = (unsigned)(ncell - c0 < 256 * kScreenCells ? ncell - c0 : 256 * kScreenCells);
  const unsigned drow = 256u / (unsigned)bx, di = 256u - drow * (unsigned)bx, dk = drow / (unsigned)by,
                 dj = drow - dk * (unsigned)by;
  int i, j, k;
  locate(c0 + tid, i, j, k);
#pragma unroll
  for (int n = 0; n < kScreenCells; ++n)
  {
    hi[n] = -1.0f;
    if (tid + n * 256u < left)
    {
      const int64_t  c = c0 + tid + n * 256;
      const double * uc = Ub + c;
      const double   u[5] = {uc[0], uc[ncell], uc[2 * ncell], uc[3 * ncell], uc[4 * ncell]};
      const double * fx = Bb + c + (j + (int64_t)by * k);
      const double * fy = Bb + nfx + c + (int64_t)bx * k;
      const double * fz = Bb + nfx + nfy + c;
      const double f[6] = {fx[0], fx[1], fy[0], fy[bx], fz[0], dim == 3 ? fz[(int64_t)bx * by] : fz[0]};
      const CflBounds b = cell_inv_dt_bounds(u, f, dim, idx, g_f, gm1, r_f, p_f, src);
      hi[n] = b.hi;
      lo = fmaxf(lo, b.lo);
    }
    i += di;
    j += dj;
    k += dk;
    if (i >= bx)
    {
      i -= bx;
      ++j;
    }
    if (j >= by)
    {
      j -= by;
      ++k;
    }
  }
  // what the CTAs before this one found is a bound too
  const double seen = __longlong_as_double((long long)*(volatile unsigned long long *)slot);
  if (seen < 1e30)
    lo = fmaxf(lo, d2f_bits(seen) * (1.0f - 2.4e-7f));
#pragma unroll
  for (int off = 16; off > 0; off >>= 1)
    lo = fmaxf(lo, __shfl_xor_sync(0xffffffffu, lo, off));
  if ((tid & 31) == 0)
    s_lo[tid >> 5] = lo;
  __syncthreads();
#pragma unroll
  for (int w = 0; w < 8; ++w)
    lo = fmaxf(lo, s_lo[w]);
  double m = 0.0;
  bool   any = false;
#pragma unroll 1
  for (int n = 0; n < kScreenCells; ++n)
  {
    const int64_t c = c0 + tid + n * 256;
    float         h = hi[0];
#pragma unroll
    for (int q = 1; q < kScreenCells; ++q)
      h = n == q ? hi[q] : h;
    if (h >= lo && c < ncell)
    {
      int i, j, k;
      locate(c, i, j, k);
      m = fmax(m, cell_inv_dt_fp64(Ub, Bb, dim, bx, by, i, j, k, c, ncell, nfx, nfy, dx_of(), gamma0, smallr, smallp, src));
      any = true;
    }
  }
  // most CTAs evaluate nothing once the slot holds a large value
  if (!__syncthreads_or(any))
    return;
#pragma unroll
  for (int off = 16; off > 0; off >>= 1)
    m = fmax(m, __shfl_xor_sync(0xffffffffu, m, off));
  if ((tid & 31) == 0)
    s_m[tid >> 5] = m;
  __syncthreads();
  if (tid == 0)
  {
    for (int w = 1; w < 8; ++w)
      m = fmax(m, s_m[w]);
    // positive doubles order like their bit patterns
    atomicMax(slot, (unsigned long long)__double_as_longlong(m));
  }
}
#endif
} // namespace gmhd
