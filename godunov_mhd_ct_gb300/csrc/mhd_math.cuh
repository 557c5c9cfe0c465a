// Per-cell MHD math on the device, templated on the compute type R (double or float).
//
// Same operand order as godunov_mhd_ct's models/mhd_utils.h and models/RiemannSolvers_MHD.h, so
// that the double instantiation, compiled with --fmad=false, gives the same bits as an FP64 host
// build of the reference formulas. Citations are to those files.
#pragma once

#include <cstdint>
#include <type_traits>

#include "exact_solvers.cuh"

namespace gmhd
{

// Variable slots (models/MHD.h:35-62): ID, IP, IU, IV, IW, IA, IB, IC.
enum : int
{
  ID = 0,
  IP = 1,
  IU = 2,
  IV = 3,
  IW = 4,
  IA = 5,
  IB = 6,
  IC = 7
};

// Riemann solver ids (models/riemann_solver_types.h:26-37).
enum : int
{
  RS_LLF = 2,
  RS_HLL = 3,
  RS_HLLC = 4,
  RS_HLLD = 5
};

// Source terms of the step (all off by default): uniform gravity and viscosity.
struct Sources
{
  int    gravity;        // [gravity] enabled
  double g[3];           // [gravity] uniform_gx, uniform_gy, uniform_gz
  int    viscosity;      // [viscosity] enabled
  double mu;             // [viscosity] mu
  int    visc_predictor; // viscous term of the Hancock predictor
};

// One cell's 1/dt from its fast speeds v_d = c_f,d + |u_d| (ComputeDtMHDFunctor.cpp:86-151): sum of
// v_d / dx; with gravity each term is scaled by k / (sqrt(1 + 2k) - 1), k = sum|g| dx / sum v_d^2
// floored at 1e-4 (:155-249); with viscosity at least 4 nu / dx^2, nu = mu / rho of the conservative
// density (:144-148). FP64 with the reference's operand order.
__device__ __forceinline__ double
cfl_inv_dt_fp64(int dim, double vx, double vy, double vz, double dx, double rho, const Sources & s)
{
  double      val;
  const Rcp64 idx = rcp64(dx);
  if (s.gravity)
  {
    double v2 = vx * vx + vy * vy;
    if (dim == 3)
      v2 += vz * vz;
    double k = fabs(s.g[0]) + fabs(s.g[1]);
    if (dim == 3)
      k += fabs(s.g[2]);
    k *= div64(dx, v2);
    k = dmax(k, 1e-4);
    const double factor = div64(k, sqrt64(1.0 + 2.0 * k) - 1.0);
    val = 0.0;
    val += div64(vx * factor, idx);
    val += div64(vy * factor, idx);
    if (dim == 3)
      val += div64(vz * factor, idx);
  }
  else
    val = dim == 3 ? div64(vx, idx) + div64(vy, idx) + div64(vz, idx) : div64(vx, idx) + div64(vy, idx);
  if (s.viscosity)
  {
    const double nu = div64(s.mu, rho);
    val = dmax(val, div64(4 * nu, dx * dx));
  }
  return val;
}

// The same from a cell's conservative state and cell-centred field: primitive recovery
// (models/mhd_utils.h:449-515), fast speeds (find_speed_info, :340-394), then cfl_inv_dt_fp64.
// Units that call it are compiled with --fmad=false, so every caller gets the same bits.
__device__ __forceinline__ double
cell_inv_dt_fp64(const double * u, double Ax, double Ay, double Az, int dim, double dx, double gamma0, double smallr,
                 double smallp, const Sources & src)
{
  const double r = dmax(u[0], smallr);
  const Rcp64  ir = rcp64(r);
  const double vx = div64(u[2], ir), vy = div64(u[3], ir), vz = div64(u[4], ir);
  const double b2 = Ax * Ax + Ay * Ay + Az * Az;
  const double eint = fma(-0.5, vx * vx + vy * vy + vz * vz, div64(fma(-0.5, b2, u[1]), ir));
  const double p = dmax((gamma0 - 1.0) * r * eint, r * smallp);
  const double c2 = div64(gamma0 * p, ir);
  const double d2 = dscale_down(div64(b2, ir) + c2, 1);
  const double dd = d2 * d2;
  const double cfx = sqrt64(d2 + sqrt64(dd - div64(c2 * Ax * Ax, ir))) + fabs(vx);
  const double cfy = sqrt64(d2 + sqrt64(dd - div64(c2 * Ay * Ay, ir))) + fabs(vy);
  const double cfz = dim == 3 ? sqrt64(d2 + sqrt64(dd - div64(c2 * Az * Az, ir))) + fabs(vz) : 0.0;
  return cfl_inv_dt_fp64(dim, cfx, cfy, cfz, dx, u[0], src);
}

// compute_cfl (scheme/ComputeDtMHDFunctor.cpp:86-151) of cell (i, j, k) of one block in the C-ABI
// layout, FP64 with the reference operand order: face B averaged to the cell centre, then the above.
// Ub / Bb point at the block's U and face arrays; c is the cell's index in the block.
__device__ __forceinline__ double
cell_inv_dt_fp64(const double * __restrict__ Ub, const double * __restrict__ Bb, int dim, int bx, int by, int i,
                 int j, int k, int64_t c, int64_t ncell, int64_t nfx, int64_t nfy, double dx, double gamma0,
                 double smallr, double smallp, const Sources & src)
{
  const double Ax = dscale_down(Bb[i + (int64_t)(bx + 1) * (j + (int64_t)by * k)] +
                                  Bb[i + 1 + (int64_t)(bx + 1) * (j + (int64_t)by * k)],
                                1);
  const double Ay = dscale_down(Bb[nfx + i + (int64_t)bx * (j + (int64_t)(by + 1) * k)] +
                                  Bb[nfx + i + (int64_t)bx * (j + 1 + (int64_t)(by + 1) * k)],
                                1);
  double Az;
  if (dim == 3)
    Az = dscale_down(Bb[nfx + nfy + i + (int64_t)bx * (j + (int64_t)by * k)] +
                       Bb[nfx + nfy + i + (int64_t)bx * (j + (int64_t)by * (k + 1))],
                     1);
  else
    Az = Bb[nfx + nfy + c];
  const double u[5] = {Ub[c], Ub[ncell + c], Ub[2 * ncell + c], Ub[3 * ncell + c], Ub[4 * ncell + c]};
  return cell_inv_dt_fp64(u, Ax, Ay, Az, dim, dx, gamma0, smallr, smallp, src);
}

// FP32 estimate of cfl_inv_dt_fp64 for the mixed path. The gravity factor is evaluated as
// (sqrt(1 + 2k) + 1) / 2, equal to k / (sqrt(1 + 2k) - 1) but without its cancellation at small k.
__device__ __forceinline__ float
cfl_inv_dt_fp32(int dim, float vx, float vy, float vz, float dx, float idx, float rho, const Sources & s)
{
  float sum = vx + vy;
  if (dim == 3)
    sum += vz;
  if (s.gravity)
  {
    float v2 = vx * vx + vy * vy;
    if (dim == 3)
      v2 += vz * vz;
    float gs = fabsf((float)s.g[0]) + fabsf((float)s.g[1]);
    if (dim == 3)
      gs += fabsf((float)s.g[2]);
    const float k = fmaxf(gs * dx / v2, 1e-4f);
    sum *= 0.5f * (sqrtf(1.0f + 2.0f * k) + 1.0f);
  }
  float val = sum * idx;
  if (s.viscosity)
    val = fmaxf(val, 4.0f * ((float)s.mu / rho) * idx * idx);
  return val;
}

template <typename R>
struct Phys
{
  R   gamma0;
  R   smallr;
  R   smallc;
  R   smallp;
  R   slope_type;
  R   entho; // 1 / (gamma0 - 1); FP64 path only
  int riemann;
};

template <typename R>
__device__ __forceinline__ R
dsqrt(R x)
{
  return sqrt64(x);
}
template <>
__device__ __forceinline__ float
dsqrt<float>(float x)
{
  return sqrtf(x);
}

template <typename R>
__device__ __forceinline__ R
rmax(R a, R b)
{
  return dmax(a, b);
}
template <>
__device__ __forceinline__ float
rmax<float>(float a, float b)
{
  return fmaxf(a, b);
}
template <typename R>
__device__ __forceinline__ R
rmin(R a, R b)
{
  return dmin(a, b);
}
template <>
__device__ __forceinline__ float
rmin<float>(float a, float b)
{
  return fminf(a, b);
}
template <typename R>
__device__ __forceinline__ R
rabs(R a)
{
  return fabs(a);
}
template <>
__device__ __forceinline__ float
rabs<float>(float a)
{
  return fabsf(a);
}
// Divisions that share a divisor. FP64 gives the reference's x / y (bit-exact parity) on the integer pipe, with
// the divisor's reciprocal computed once; the FP32 path multiplies by one reciprocal inv = recip(y).
template <typename R>
__device__ __forceinline__ auto
recip(R y)
{
  if constexpr (std::is_same<R, double>::value)
    return rcp64(y);
  else
    return R(1) / y;
}
template <typename R, typename I>
__device__ __forceinline__ R
qdiv(R x, R y, const I & inv)
{
  (void)y;
  if constexpr (std::is_same<R, double>::value)
    return div64(x, inv);
  else
    return x * inv;
}
// x / y as written
template <typename R>
__device__ __forceinline__ R
rdiv(R x, R y)
{
  if constexpr (std::is_same<R, double>::value)
    return div64(x, y);
  else
    return x / y;
}
// q + 0.5 s and q - 0.5 s (0.5 s is exact, so FP64 takes one fused instruction)
template <typename R>
__device__ __forceinline__ R
plus_half(R q, R s)
{
  if constexpr (std::is_same<R, double>::value)
    return fma(0.5, s, q);
  else
    return q + R(0.5) * s;
}
template <typename R>
__device__ __forceinline__ R
minus_half(R q, R s)
{
  if constexpr (std::is_same<R, double>::value)
    return fma(-0.5, s, q);
  else
    return q + R(-0.5) * s;
}
// x / 2
template <typename R>
__device__ __forceinline__ R
half_of(R x)
{
  if constexpr (std::is_same<R, double>::value)
    return dscale_down(x, 1);
  else
    return R(0.5) * x;
}

// find_speed_fast<dir> (models/mhd_utils.h:93-122)
template <typename R>
__device__ __forceinline__ R
speed_fast(const R * q, int dir, const Phys<R> & s)
{
  const R d = q[ID], p = q[IP], a = q[IA], b = q[IB], c = q[IC];
  const auto id = recip<R>(d);
  const R b2 = a * a + b * b + c * c;
  const R c2 = qdiv<R>(s.gamma0 * p, d, id);
  const R d2 = R(0.5) * (qdiv<R>(b2, d, id) + c2);
  const R bn = dir == 0 ? a : (dir == 1 ? b : c);
  return dsqrt<R>(d2 + dsqrt<R>(d2 * d2 - qdiv<R>(c2 * bn * bn, d, id)));
}

// find_mhd_flux (models/mhd_utils.h:182-245), cIso == 0
template <typename R>
__device__ __forceinline__ void
mhd_flux(const R * q, R * cv, R * ff, const Phys<R> & s)
{
  const R p = q[IP];
  const R entho = R(1) / (s.gamma0 - R(1));
  const R d = q[ID], u = q[IU], v = q[IV], w = q[IW], a = q[IA], b = q[IB], c = q[IC];
  const R ecin = R(0.5) * (u * u + v * v + w * w) * d;
  const R emag = R(0.5) * (a * a + b * b + c * c);
  const R etot = p * entho + ecin + emag;
  const R ptot = p + emag;
  cv[ID] = d;
  cv[IP] = etot;
  cv[IU] = d * u;
  cv[IV] = d * v;
  cv[IW] = d * w;
  cv[IA] = a;
  cv[IB] = b;
  cv[IC] = c;
  ff[ID] = d * u;
  ff[IP] = (etot + ptot) * u - a * (a * u + b * v + c * w);
  ff[IU] = d * u * u - a * a + ptot;
  ff[IV] = d * u * v - a * b;
  ff[IW] = d * u * w - a * c;
  ff[IA] = R(0);
  ff[IB] = b * u - a * v;
  ff[IC] = c * u - a * w;
}

// riemann_hll (models/RiemannSolvers_MHD.h:43-102)
template <typename R>
__device__ void
riemann_hll(R * qL, R * qR, R * flux, const Phys<R> & s)
{
  const R bx_mean = R(0.5) * (qL[IA] + qR[IA]);
  qL[IA] = bx_mean;
  qR[IA] = bx_mean;
  R uL[8], fL[8], uR[8], fR[8];
  mhd_flux(qL, uL, fL, s);
  mhd_flux(qR, uR, fR, s);
  const R cfL = speed_fast(qL, 0, s);
  const R cfR = speed_fast(qR, 0, s);
  const R vL = qL[IU], vR = qR[IU];
  const R sl = rmin<R>(rmin<R>(vL, vR) - rmax<R>(cfL, cfR), R(0));
  const R sr = rmax<R>(rmax<R>(vL, vR) + rmax<R>(cfL, cfR), R(0));
#pragma unroll
  for (int n = 0; n < 8; ++n)
    flux[n] = rdiv<R>(sr * fL[n] - sl * fR[n] + sr * sl * (uR[n] - uL[n]), sr - sl);
}

// riemann_llf (models/RiemannSolvers_MHD.h:118-153)
template <typename R>
__device__ void
riemann_llf(R * qL, R * qR, R * flux, const Phys<R> & s)
{
  const R bx_mean = R(0.5) * (qL[IA] + qR[IA]);
  qL[IA] = bx_mean;
  qR[IA] = bx_mean;
  R uL[8], fL[8], uR[8], fR[8];
  mhd_flux(qL, uL, fL, s);
  mhd_flux(qR, uR, fR, s);
#pragma unroll
  for (int n = 0; n < 8; ++n)
    flux[n] = (fL[n] + fR[n]) / R(2);
  // x-direction info speed (models/mhd_utils.h:405-433)
  R cinfo[2];
  for (int side = 0; side < 2; ++side)
  {
    const R * q = side == 0 ? qL : qR;
    const R   d = q[ID], p = q[IP], a = q[IA], b = q[IB], c = q[IC];
    const R   b2 = a * a + b * b + c * c;
    const R   c2 = s.gamma0 * p / d;
    const R   d2 = R(0.5) * (b2 / d + c2);
    const R   cf = dsqrt<R>(d2 + dsqrt<R>(d2 * d2 - c2 * a * a / d));
    cinfo[side] = cf + rabs<R>(q[IU]);
  }
  const R vel_info = rmax<R>(cinfo[0], cinfo[1]);
#pragma unroll
  for (int n = 0; n < 8; ++n)
    flux[n] -= vel_info * (uR[n] - uL[n]) / R(2);
}

// riemann_hllc (models/RiemannSolvers_MHD.h:165-286); components IA..IC are left at 0
template <typename R>
__device__ void
riemann_hllc(const R * qL, const R * qR, R * flux, const Phys<R> & s)
{
  const R entho = R(1) / (s.gamma0 - R(1));
  const R rl = rmax<R>(qL[ID], s.smallr);
  const R pl = rmax<R>(qL[IP], rl * s.smallp);
  const R ul = qL[IU];
  R       ecinl = R(0.5) * rl * ul * ul;
  ecinl += R(0.5) * rl * qL[IV] * qL[IV];
  ecinl += R(0.5) * rl * qL[IW] * qL[IW];
  const R etotl = pl * entho + ecinl;
  const R ptotl = pl;
  const R rr = rmax<R>(qR[ID], s.smallr);
  const R pr = rmax<R>(qR[IP], rr * s.smallp);
  const R ur = qR[IU];
  R       ecinr = R(0.5) * rr * ur * ur;
  ecinr += R(0.5) * rr * qR[IV] * qR[IV];
  ecinr += R(0.5) * rr * qR[IW] * qR[IW];
  const R etotr = pr * entho + ecinr;
  const R ptotr = pr;
  const R cfastl = dsqrt<R>(rmax<R>(s.gamma0 * pl / rl, s.smallc * s.smallc));
  const R cfastr = dsqrt<R>(rmax<R>(s.gamma0 * pr / rr, s.smallc * s.smallc));
  const R SL = rmin<R>(ul, ur) - rmax<R>(cfastl, cfastr);
  const R SR = rmax<R>(ul, ur) + rmax<R>(cfastl, cfastr);
  const R rcl = rl * (ul - SL);
  const R rcr = rr * (SR - ur);
  const R ustar = (rcr * ur + rcl * ul + (ptotl - ptotr)) / (rcr + rcl);
  const R ptotstar = (rcr * ptotl + rcl * ptotr + rcl * rcr * (ul - ur)) / (rcr + rcl);
  const R rstarl = rl * (SL - ul) / (SL - ustar);
  const R etotstarl = ((SL - ul) * etotl - ptotl * ul + ptotstar * ustar) / (SL - ustar);
  const R rstarr = rr * (SR - ur) / (SR - ustar);
  const R etotstarr = ((SR - ur) * etotr - ptotr * ur + ptotstar * ustar) / (SR - ustar);
  R       ro, uo, ptoto, etoto;
  if (SL > R(0))
  {
    ro = rl; uo = ul; ptoto = ptotl; etoto = etotl;
  }
  else if (ustar > R(0))
  {
    ro = rstarl; uo = ustar; ptoto = ptotstar; etoto = etotstarl;
  }
  else if (SR > R(0))
  {
    ro = rstarr; uo = ustar; ptoto = ptotstar; etoto = etotstarr;
  }
  else
  {
    ro = rr; uo = ur; ptoto = ptotr; etoto = etotr;
  }
  flux[ID] = ro * uo;
  flux[IU] = ro * uo * uo + ptoto;
  flux[IP] = (etoto + ptoto) * uo;
  flux[IV] = flux[ID] > R(0) ? flux[ID] * qL[IV] : flux[ID] * qR[IV];
  flux[IW] = flux[ID] > R(0) ? flux[ID] * qL[IW] : flux[ID] * qR[IW];
}

// ---- mixed path: HLLD fluxes and edge EMFs with every FP32 rounding written out -------------------------------
// Which product of a sum like a b + c d is fused into an FMA is the compiler's choice, and it chose differently from one
// tile's kernel to another (and from one edit to the next): results of the mixed path then differ in the last FP32
// bits. The two solvers below name each operation, so that a kernel's bits do not change with the code around them. The edge
// solver rounds alike in every kernel; HLLD keeps the three forms that the kernels had (below).
__device__ __forceinline__ float
fmul_(float a, float b)
{
  return __fmul_rn(a, b);
}
__device__ __forceinline__ float
fadd_(float a, float b)
{
  return __fadd_rn(a, b);
}
// a b + c d and a b - c d, the first product fused
__device__ __forceinline__ float
sum2(float a, float b, float c, float d)
{
  return __fmaf_rn(a, b, __fmul_rn(c, d));
}
__device__ __forceinline__ float
dif2(float a, float b, float c, float d)
{
  return __fmaf_rn(a, b, -__fmul_rn(c, d));
}

// v + g dt / 2; FP32 with the product fused with the addition or not, as each kernel has always had it (Cfg::KICK_FUSED)
template <typename R, bool FUSED>
__device__ __forceinline__ R
half_kick(R v, R g, R dt)
{
  if constexpr (std::is_same<R, double>::value)
    return v + g * 0.5 * dt;
  else if constexpr (FUSED)
    return __fmaf_rn(0.5f * g, dt, v);
  else
    return fadd_(v, fmul_(0.5f * g, dt));
}

// The rounding of r (S - u)^2 - a^2 on the left and right side (e): the product fused with the subtraction or not, as each
// kernel has always had it (Cfg::hlld_fuse). No form is more accurate than the others by more than an FP32 rounding.
enum : int
{
  HLLD_PLAIN = 0,  // neither
  HLLD_FUSE_R = 1, // right side
  HLLD_FUSE_LR = 3 // both
};

// riemann_hlld (models/RiemannSolvers_MHD.h:311-551), Miyoshi & Kusano 2005, of two states with the normal field a. The
// FP64 path's: riemann_hlld_fp64.
template <int FUSE>
__device__ __forceinline__ void
riemann_hlld_f32(const float * qL, const float * qR, float a, float * flux, const Phys<float> & s)
{
  const float entho = 1.0f / (s.gamma0 - 1.0f);
  const float sgnm = (a >= 0) ? 1.0f : -1.0f;
  const float aa = fmul_(a, a);
  float       et[2], pt[2], vb[2], cf[2];
#pragma unroll
  for (int k = 0; k < 2; ++k)
  {
    const float * q = k ? qR : qL;
    const float   r = q[ID], p = q[IP], u = q[IU], v = q[IV], w = q[IW], b = q[IB], c = q[IC];
    const float   kin = fmul_(0.5f, __fmaf_rn(w, w, sum2(u, u, v, v)));
    const float   b2 = __fmaf_rn(c, c, __fmaf_rn(b, b, aa));
    et[k] = __fmaf_rn(0.5f, b2, sum2(p, entho, kin, r));
    pt[k] = __fmaf_rn(0.5f, b2, p);
    vb[k] = __fmaf_rn(w, c, sum2(u, a, v, b));
    // find_speed_fast
    const float id = 1.0f / r;
    const float gp = fmul_(s.gamma0, p), c2 = fmul_(gp, id);
    const float d2 = fmul_(0.5f, sum2(b2, id, gp, id));
    cf[k] = sqrtf(fadd_(d2, sqrtf(dif2(d2, d2, fmul_(fmul_(c2, a), a), id))));
  }
  const float rl = qL[ID], ul = qL[IU], rr = qR[ID], ur = qR[IU];
  const float cm = fmaxf(cf[0], cf[1]);
  const float sl = fadd_(fminf(ul, ur), -cm), sr = fadd_(fmaxf(ul, ur), cm);
  const float rcl = fmul_(rl, fadd_(ul, -sl)), rcr = fmul_(rr, fadd_(sr, -ur));
  const float irc = 1.0f / fadd_(rcr, rcl);
  const float us = fmul_(fadd_(sum2(rcr, ur, rcl, ul), fadd_(pt[0], -pt[1])), irc);
  const float ps = fmul_(__fmaf_rn(fmul_(rcl, rcr), fadd_(ul, -ur), sum2(rcr, pt[0], rcl, pt[1])), irc);
  const float psus = fmul_(ps, us), ua = fmul_(us, a);
  // star states
  float rs[2], vs[2], ws[2], bs[2], cs[2], vbs[2], es[2], sq[2], sa[2];
#pragma unroll
  for (int k = 0; k < 2; ++k)
  {
    const float * q = k ? qR : qL;
    const float   r = q[ID], u = q[IU], v = q[IV], w = q[IW], b = q[IB], c = q[IC];
    const float   m = fadd_(k ? sr : sl, -u), n = fadd_(k ? sr : sl, -us);
    const float   in = 1.0f / n;
    const float   rm = fmul_(r, m);
    rs[k] = fmul_(rm, in);
    const float estar = dif2(rm, n, a, a);
    const float e = ((FUSE >> (1 - k)) & 1) ? __fmaf_rn(rm, m, -aa) : fadd_(fmul_(rm, m), -aa);
    if (fabsf(estar) < 1e-4f * aa)
    {
      vs[k] = v;
      bs[k] = b;
      ws[k] = w;
      cs[k] = c;
    }
    else
    {
      const float ie = 1.0f / estar, du = fadd_(us, -u);
      vs[k] = __fmaf_rn(-fmul_(fmul_(a, b), du), ie, v);
      bs[k] = fmul_(fmul_(b, e), ie);
      ws[k] = __fmaf_rn(-fmul_(fmul_(a, c), du), ie, w);
      cs[k] = fmul_(fmul_(c, e), ie);
    }
    vbs[k] = __fmaf_rn(ws[k], cs[k], __fmaf_rn(vs[k], bs[k], ua));
    es[k] = fmul_(__fmaf_rn(a, fadd_(vb[k], -vbs[k]), fadd_(psus, dif2(m, et[k], pt[k], u))), in);
    const float rq = rsqrtf(rs[k]);
    sq[k] = fmul_(rs[k], rq);
    sa[k] = __fmaf_rn(k ? fabsf(a) : -fabsf(a), rq, us);
  }
  const float isq = 1.0f / fadd_(sq[0], sq[1]);
  const float vss = fmul_(__fmaf_rn(sgnm, fadd_(bs[1], -bs[0]), sum2(sq[0], vs[0], sq[1], vs[1])), isq);
  const float wss = fmul_(__fmaf_rn(sgnm, fadd_(cs[1], -cs[0]), sum2(sq[0], ws[0], sq[1], ws[1])), isq);
  const float s0 = fmul_(sgnm, sq[0]), qq = fmul_(s0, sq[1]);
  const float bss = fmul_(__fmaf_rn(qq, fadd_(vs[1], -vs[0]), sum2(sq[0], bs[1], sq[1], bs[0])), isq);
  const float css = fmul_(__fmaf_rn(qq, fadd_(ws[1], -ws[0]), sum2(sq[0], cs[1], sq[1], cs[0])), isq);
  const float vbss = __fmaf_rn(wss, css, __fmaf_rn(vss, bss, ua));
  const float essl = fadd_(es[0], -fmul_(s0, fadd_(vbs[0], -vbss)));
  const float essr = __fmaf_rn(fmul_(sgnm, sq[1]), fadd_(vbs[1], -vbss), es[1]);

  // the state on the face, in the order sl, sal, ustar, sar, sr > 0: its side, and whether outside the fan, between
  // the fast and the Alfven wave (star) or between that and the contact
  const bool  left = sl > 0 || sa[0] > 0 || us > 0;
  const bool  outer = left ? sl > 0 : !(sa[1] > 0 || sr > 0);
  const bool  inner = left ? !(sa[0] > 0) : sa[1] > 0;
  const float ro = outer ? (left ? rl : rr) : (left ? rs[0] : rs[1]);
  const float uo = outer ? (left ? ul : ur) : us;
  const float vo = outer ? (left ? qL[IV] : qR[IV]) : (inner ? vss : (left ? vs[0] : vs[1]));
  const float wo = outer ? (left ? qL[IW] : qR[IW]) : (inner ? wss : (left ? ws[0] : ws[1]));
  const float bo = outer ? (left ? qL[IB] : qR[IB]) : (inner ? bss : (left ? bs[0] : bs[1]));
  const float co = outer ? (left ? qL[IC] : qR[IC]) : (inner ? css : (left ? cs[0] : cs[1]));
  const float po = outer ? (left ? pt[0] : pt[1]) : ps;
  const float eo = outer ? (left ? et[0] : et[1]) : (inner ? (left ? essl : essr) : (left ? es[0] : es[1]));
  const float vbo = outer ? (left ? vb[0] : vb[1]) : (inner ? vbss : (left ? vbs[0] : vbs[1]));
  const float ru = fmul_(ro, uo);
  flux[ID] = ru;
  flux[IP] = dif2(fadd_(eo, po), uo, a, vbo);
  flux[IU] = fadd_(dif2(ru, uo, a, a), po);
  flux[IV] = dif2(ru, vo, a, bo);
  flux[IW] = dif2(ru, wo, a, co);
  flux[IA] = 0.0f;
  flux[IB] = dif2(bo, uo, a, vo);
  flux[IC] = dif2(co, uo, a, wo);
}

// riemann_mhd dispatch (models/RiemannSolvers_MHD.h:559-590); both states hold the face's normal field in IA
template <typename R, int FUSE = HLLD_PLAIN>
__device__ __forceinline__ void
riemann_mhd(R * qL, R * qR, R * flux, const Phys<R> & s)
{
  if (s.riemann == RS_HLLD)
  {
    if constexpr (std::is_same<R, double>::value)
      riemann_hlld_fp64(qL, qR, flux, s.gamma0, s.entho);
    else
      riemann_hlld_f32<FUSE>(qL, qR, qL[IA], flux, s);
  }
  else if (s.riemann == RS_HLL)
    riemann_hll(qL, qR, flux, s);
  else if (s.riemann == RS_LLF)
    riemann_llf(qL, qR, flux, s);
  else
  {
#pragma unroll
    for (int n = 0; n < 8; ++n)
      flux[n] = R(0);
    riemann_hllc(qL, qR, flux, s);
  }
}

// The scheme's maxima of several values, r = x0; r = x > r ? x : r for the others (a NaN first value stays, another
// is passed over), with three-input maxima and one comparison
__device__ __forceinline__ float
max4(float x0, float x1, float x2, float x3)
{
  const float m = fmaxf(fmaxf(x1, x2), x3);
  return m > x0 ? m : x0;
}
__device__ __forceinline__ float
min4(float x0, float x1, float x2, float x3)
{
  const float m = fminf(fminf(x1, x2), x3);
  return m < x0 ? m : x0;
}
__device__ __forceinline__ float
max5(float x0, float x1, float x2, float x3, float x4)
{
  const float m = fmaxf(fmaxf(fmaxf(x1, x2), x3), x4);
  return m > x0 ? m : x0;
}

// Edge-state slots: reconstructed states around an edge.
enum : int
{
  ERT = 0,
  ELT = 1,
  ERB = 2,
  ELB = 3
};

// compute_emf<dir> + mag_riemann2d_hlld (models/RiemannSolvers_MHD.h:629-869, 890-1097) of the mixed path (FP64:
// edge_emf_fp64). The four states around the edge in the order LL, LR, RL, RR: density, pressure, velocities u, v and
// orthogonal field c; the transverse field is shared, a0 by LL and RL, a1 by LR and RR, b0 by LL and LR, b1 by RL and RR
// (the scheme averages two equal values, except By on x edges). Of the nine wave-fan regions' terms all but one have
// weight 0: only the common region's is always computed. With the three-input maxima this is 100 of 786 instructions
// an edge less: 256^3 6.43 -> 6.05 ms a step, 96 field loops 8.20 -> 7.72 ms for ten steps.
__device__ __forceinline__ float
edge_emf_f32(const float * r, const float * p, const float * u, const float * v, const float * c, float a0, float a1,
             float b0, float b1, const Phys<float> & s)
{
  const float a[4] = {a0, a1, a0, a1}, b[4] = {b0, b0, b1, b1};
  float       fx[4], fy[4], pt[4];
#pragma unroll
  for (int k = 0; k < 4; ++k)
  {
    // find_speed_fast along both axes
    const float id = 1.0f / r[k];
    const float b2 = __fmaf_rn(c[k], c[k], sum2(a[k], a[k], b[k], b[k]));
    const float gp = fmul_(s.gamma0, p[k]), c2 = fmul_(gp, id);
    const float d2 = fmul_(0.5f, sum2(b2, id, gp, id)), dd = fmul_(d2, d2);
    fx[k] = sqrtf(fadd_(d2, sqrtf(__fmaf_rn(-fmul_(fmul_(c2, a[k]), a[k]), id, dd))));
    fy[k] = sqrtf(fadd_(d2, sqrtf(__fmaf_rn(-fmul_(fmul_(c2, b[k]), b[k]), id, dd))));
    pt[k] = __fmaf_rn(0.5f, b2, p[k]);
  }
  const float cx = max4(fx[0], fx[1], fx[2], fx[3]), cy = max4(fy[0], fy[1], fy[2], fy[3]);
  const float SL = fadd_(min4(u[0], u[1], u[2], u[3]), -cx), SR = fadd_(max4(u[0], u[1], u[2], u[3]), cx);
  const float SB = fadd_(min4(v[0], v[1], v[2], v[3]), -cy), ST = fadd_(max4(v[0], v[1], v[2], v[3]), cy);
  const float rx0 = fmul_(r[0], fadd_(u[0], -SL)), rx1 = fmul_(r[1], fadd_(u[1], -SL));
  const float rx2 = fmul_(r[2], fadd_(SR, -u[2])), rx3 = fmul_(r[3], fadd_(SR, -u[3]));
  const float ry0 = fmul_(r[0], fadd_(v[0], -SB)), ry1 = fmul_(r[1], fadd_(ST, -v[1]));
  const float ry2 = fmul_(r[2], fadd_(v[2], -SB)), ry3 = fmul_(r[3], fadd_(ST, -v[3]));
  const float ustar = fadd_(__fmaf_rn(rx3, u[3], __fmaf_rn(rx2, u[2], sum2(rx0, u[0], rx1, u[1]))),
                            fadd_(fadd_(fadd_(pt[0], -pt[2]), pt[1]), -pt[3])) /
                      fadd_(fadd_(fadd_(rx0, rx1), rx2), rx3);
  const float vstar = fadd_(__fmaf_rn(ry3, v[3], __fmaf_rn(ry2, v[2], sum2(ry0, v[0], ry1, v[1]))),
                            fadd_(fadd_(fadd_(pt[0], -pt[1]), pt[2]), -pt[3])) /
                      fadd_(fadd_(fadd_(ry0, ry1), ry2), ry3);
  const float iL = 1.0f / fadd_(SL, -ustar), iR = 1.0f / fadd_(SR, -ustar);
  const float iB = 1.0f / fadd_(SB, -vstar), iT = 1.0f / fadd_(ST, -vstar);
  float       As[4], Bs[4], qx[4], qy[4], qs[4]; // star fields; densities past the x wave, the y wave and both
#pragma unroll
  for (int k = 0; k < 4; ++k)
  {
    const float X = fadd_(k & 2 ? SR : SL, -u[k]), Y = fadd_(k & 1 ? ST : SB, -v[k]);
    const float ix = k & 2 ? iR : iL, iy = k & 1 ? iT : iB;
    qx[k] = fmul_(fmul_(r[k], X), ix);
    Bs[k] = fmul_(fmul_(b[k], X), ix);
    qy[k] = fmul_(fmul_(r[k], Y), iy);
    As[k] = fmul_(fmul_(a[k], Y), iy);
    qs[k] = fmul_(fmul_(qx[k], Y), iy);
  }
  auto        al = [](float f, float q) { return fmul_(fabsf(f), rsqrtf(q)); };
  const float cL = max5(al(a1, qx[1]), al(As[1], qs[1]), al(a0, qx[0]), al(As[0], qs[0]), s.smallc);
  const float cR = max5(al(a1, qx[3]), al(As[3], qs[3]), al(a0, qx[2]), al(As[2], qs[2]), s.smallc);
  const float cB = max5(al(b0, qy[0]), al(Bs[0], qs[0]), al(b1, qy[2]), al(Bs[2], qs[2]), s.smallc);
  const float cT = max5(al(b0, qy[1]), al(Bs[1], qs[1]), al(b1, qy[3]), al(Bs[3], qs[3]), s.smallc);
  const float SAL = fminf(fadd_(ustar, -cL), 0.0f), SAR = fmaxf(fadd_(ustar, cR), 0.0f);
  const float SAB = fminf(fadd_(vstar, -cB), 0.0f), SAT = fmaxf(fadd_(vstar, cT), 0.0f);
  const float iRL = 1.0f / fadd_(SAR, -SAL), iTB = 1.0f / fadd_(SAT, -SAB);
  const float LB = fmul_(SAL, SAB), LT = fmul_(SAL, SAT), RB = fmul_(SAR, SAB), RT = fmul_(SAR, SAT);
  const float TB = fmul_(SAT, SAB), RL = fmul_(SAR, SAL);
  auto        es = [&](int k) { return dif2(ustar, Bs[k], vstar, As[k]); };
  const float sum = __fmaf_rn(RT, es(0), __fmaf_rn(-RB, es(1), dif2(LB, es(3), LT, es(2))));
  const float dA = dif2(dif2(SAR, As[3], SAL, As[1]), iRL, dif2(SAR, As[2], SAL, As[0]), iRL);
  const float dB = dif2(dif2(SAT, Bs[3], SAB, Bs[2]), iTB, dif2(SAT, Bs[1], SAB, Bs[0]), iTB);
  const float mid = __fmaf_rn(fmul_(RL, iRL), dB, dif2(fmul_(sum, iRL), iTB, fmul_(TB, iTB), dA));
  // the fan spans the edge along both axes: the one region with weight 1
  const bool sbn = __float_as_int(SB) < 0, stn = __float_as_int(ST) < 0, sln = __float_as_int(SL) < 0, srn = __float_as_int(SR) < 0;
  if (sbn && !stn && sln && !srn)
    return mid;
  const float sbp = sbn ? 0.0f : 1.0f, stp = stn ? 0.0f : 1.0f, slp = sln ? 0.0f : 1.0f, srp = srn ? 0.0f : 1.0f;
  const float sbm = 1.0f - sbp, stm = 1.0f - stp, slm = 1.0f - slp, srm = 1.0f - srp;
  auto        e0 = [&](int k) { return dif2(u[k], b[k], v[k], a[k]); };
  auto        ex = [&](int k) { return dif2(ustar, Bs[k], v[k], a[k]); };
  auto        ey = [&](int k) { return dif2(u[k], b[k], vstar, As[k]); };
  auto        along_x = [&](int k) { // bottom (k = 0) and top (k = 1)
    const float t = fmul_(__fmaf_rn(RL, fadd_(b1, -b0), dif2(SAR, ex(k), SAL, ex(k + 2))), iRL);
    return slp * e0(k) + slm * srm * e0(k + 2) + slm * srp * t;
  };
  auto along_y = [&](int k) { // left (k = 0) and right (k = 2)
    return fmul_(__fmaf_rn(-TB, fadd_(a1, -a0), dif2(SAT, ey(k), SAB, ey(k + 1))), iTB);
  };
  float E = (sbm * stp * slm * srp) * mid;
  E += sbp * along_x(0);
  E += (sbm * stm) * along_x(1);
  E += (sbm * stp * slp) * along_y(0);
  E += (sbm * stp * slm * srm) * along_y(2);
  return E;
}

// EMF along CD from the reconstructed states qe[ERT..ELB]
template <int CD, int DIM>
__device__ __forceinline__ float
edge_emf(const float (*qe)[8], const Phys<float> & s)
{
  // (u, v) and (a, b) the edge's transverse axes in turn, c along it
  constexpr int  iu = CD == 2 ? IU : (CD == 1 ? IW : IV), iv = CD == 2 ? IV : (CD == 1 ? IU : IW);
  constexpr int  ia = iu + 3, ib = iv + 3, ic = CD == 2 ? IC : (CD == 1 ? IB : IA);
  constexpr bool own = DIM == 3 && CD == 0; // By on x edges: the scheme adds each cell's own slopes to the face's
  const float *  st[4] = {qe[ERT], qe[ERB], qe[ELT], qe[ELB]};
  float          r[4], p[4], u[4], v[4], c[4];
#pragma unroll
  for (int q = 0; q < 4; ++q)
  {
    r[q] = st[q][ID];
    p[q] = st[q][IP];
    u[q] = st[q][iu];
    v[q] = st[q][iv];
    c[q] = st[q][ic];
  }
  const float a0 = own ? half_of<float>(qe[ERT][ia] + qe[ELT][ia]) : qe[ERT][ia];
  const float a1 = own ? half_of<float>(qe[ERB][ia] + qe[ELB][ia]) : qe[ERB][ia];
  return edge_emf_f32(r, p, u, v, c, a0, a1, qe[ERT][ib], qe[ELT][ib], s);
}

// slope_unsplit_scalar (scheme/ComputeLimitedSlopesFunctor.cpp:121-144)
template <typename R>
__device__ __forceinline__ R
slope1(R q, R qp, R qm, R slope_type)
{
  if constexpr (std::is_same<R, double>::value)
    return slope1_fp64(q, qp, qm, slope_type);
  R dq = 0;
  if (slope_type == R(1) || slope_type == R(2))
  {
    const R dlft = slope_type * (q - qm);
    const R drgt = slope_type * (qp - q);
    const R dcen = R(0.5) * (qp - qm);
    const R dsgn = (dcen >= R(0)) ? R(1) : R(-1);
    const R slop = rmin<R>(rabs<R>(dlft), rabs<R>(drgt));
    const R dlim = (dlft * drgt) <= R(0) ? R(0) : slop;
    dq = dsgn * rmin<R>(dlim, rabs<R>(dcen));
  }
  return dq;
}

} // namespace gmhd

namespace gmhd
{
// FP64 <-> FP32 conversions on the integer pipe. On GB300 the FP64 pipe (which also executes
// F2F conversions) has a small fraction of the FP32 rate, so the mixed path converts by
// rebuilding the IEEE-754 bit patterns instead.

// double -> float, rounding the 29 dropped mantissa bits half away from zero; results below the
// float normal range flush to signed zero, above it saturate to infinity; NaN stays NaN.
__device__ __forceinline__ float
d2f_bits(double x)
{
  const unsigned hi = (unsigned)__double2hiint(x);
  const unsigned lo = (unsigned)__double2loint(x);
  const unsigned sign = hi & 0x80000000u;
  const unsigned mag = hi & 0x7fffffffu;
  // the low 8 exponent bits and the top 23 mantissa bits in place (one funnel shift); for exponents
  // 897..1150 (the float normal range) e - 896 == (e & 0xff) ^ 0x80, so the rebias 1023 -> 127 is a
  // flip of the field's top bit; then the first dropped bit rounds, a carry out of the mantissa
  // moving into the exponent as it should
  const unsigned bits = ((__funnelshift_l(lo, hi, 3) & 0x7fffffffu) ^ 0x40000000u) + ((lo >> 28) & 1u);
  // |x| below the float normal range (exponent <= 896) -> signed zero; at or above 2^128
  // (exponent >= 1151), infinity or NaN -> infinity / quiet NaN
  if (mag < 0x38100000u)
    return __uint_as_float(sign);
  if (mag >= 0x47f00000u)
  {
    const bool nan = mag > 0x7ff00000u || (mag == 0x7ff00000u && lo != 0u);
    return __uint_as_float(sign | 0x7f800000u | (nan ? 0x400000u : 0u));
  }
  return __uint_as_float(sign | bits);
}

// float -> double, exact for normal numbers, zero, infinity and NaN (subnormals flush to zero).
__device__ __forceinline__ double
f2d_bits(float x)
{
  const unsigned b = __float_as_uint(x);
  const unsigned sign = b & 0x80000000u;
  const unsigned e = (b >> 23) & 0xffu;
  const unsigned m = b & 0x7fffffu;
  const unsigned eb = e == 0xffu ? 0x7ffu : e + 896u;
  unsigned       hi = sign | (eb << 20) | (m >> 3);
  unsigned       lo = m << 29;
  hi = e == 0u ? sign : hi;
  lo = e == 0u ? 0u : lo;
  return __hiloint2double((int)hi, (int)lo);
}

// Adds t to the running sum s and the rounding error of that addition to e (Knuth's TwoSum: six
// FP32 operations, no branch, valid for any magnitudes; no multiply, so FMA contraction cannot
// change it). After the last term, s + e holds the exact sum of the terms up to the rounding of e
// itself, which is of order eps^2 relative to the terms.
__device__ __forceinline__ void
two_sum_acc(float & s, float & e, float t)
{
  const float u = s + t;
  const float tb = u - s;
  const float err = (s - (u - tb)) + (t - tb);
  s = u;
  e += err;
}

template <typename R>
__device__ __forceinline__ R
to_r(double x)
{
  return x;
}
template <>
__device__ __forceinline__ float
to_r<float>(double x)
{
  return d2f_bits(x);
}

template <typename R>
__device__ __forceinline__ double
to_d(R x)
{
  return x;
}
template <>
__device__ __forceinline__ double
to_d<float>(float x)
{
  return f2d_bits(x);
}
} // namespace gmhd
