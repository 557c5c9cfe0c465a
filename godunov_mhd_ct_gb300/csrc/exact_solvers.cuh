// FP64 slopes, HLLD fluxes and edge EMFs of the exact path: the values of the templates in mhd_math.cuh, bit for
// bit, with as few FP64 instructions as the operand order allows.
//
// What bounds the exact path is the FP64 pipe (two lanes per SM and clock). Divisions and square roots run on the
// integer pipe (fp64_int.cuh), and so do comparisons, signs, minima and scalings by powers of two; q + 0.5 s is one fused
// multiply-add (0.5 s is exact). Where the scheme takes the largest of several speeds, FP32 estimates of their
// differences show which can be the largest: only those are evaluated in FP64 (one of four fast speeds, one of four
// Alfven speeds a side; all of them, in the scheme's order, where the estimates are unusable). The weights 0 and 1 of
// the EMF's nine wave-fan regions become a branch on the region.
// 3D Orszag-Tang 128^3, FP64: 42.3 -> 15.0 ms a step; 2D 128^2: 315 -> 82 us. The FP64 pipe is still what bounds it
// (68 % busy at 16.5 ms), now with the scheme's additions and multiplications.
#pragma once

#include "fp64_int.cuh"

namespace gmhd
{

GMHD_CALL double
slow_slope(double q, double qp, double qm, double st)
{
  const double dlft = st * (q - qm);
  const double drgt = st * (qp - q);
  const double dcen = 0.5 * (qp - qm);
  const double dsgn = (dcen >= 0.0) ? 1.0 : -1.0;
  const double slop = fmin(fabs(dlft), fabs(drgt));
  const double dlim = (dlft * drgt) <= 0.0 ? 0.0 : slop;
  return dsgn * fmin(dlim, fabs(dcen));
}

// slope_unsplit_scalar (scheme/ComputeLimitedSlopesFunctor.cpp:121-144) with three FP64 subtractions: the products
// with slope_type (1 or 2) and 0.5 are exponent shifts, the sign test and the minima integer ones
__device__ __forceinline__ double
slope1_fp64(double q, double qp, double qm, double st)
{
  const int64_t stb = (int64_t)__double_as_longlong(st);
  if (stb != 0x3ff0000000000000ll && stb != 0x4000000000000000ll)
    return 0.0;
  const uint64_t a = (uint64_t)__double_as_longlong(q - qm), b = (uint64_t)__double_as_longlong(qp - q),
                 c = (uint64_t)__double_as_longlong(qp - qm);
  const uint64_t mask = 0x7fffffffffffffffull;
  const uint64_t ma = a & mask, mb = b & mask, mc = c & mask;
  const bool     zero = (int64_t)(a ^ b) < 0 || ma == 0u || mb == 0u;
  uint64_t       lo = ma < mb ? ma : mb;
  const uint32_t ha = (uint32_t)(ma >> 32), hb = (uint32_t)(mb >> 32), hc = (uint32_t)(mc >> 32);
  uint32_t       top = ha > hb ? ha : hb;
  top = top > hc ? top : hc;
  // differences below 2^-523 or close to overflow, infinities and NaN
  if (top >= 0x7fe00000u || (!zero && (uint32_t)(lo >> 32) < 0x1f400000u))
    return slow_slope(q, qp, qm, st);
  lo += stb == 0x4000000000000000ll ? 0x0010000000000000ull : 0ull;
  const uint64_t h = mc - 0x0010000000000000ull;
  lo = lo < h ? lo : h;
  lo = zero ? 0u : lo;
  return __longlong_as_double((long long)(lo | (c & ~mask)));
}

// |x| in FP32, truncated (within 2^-23); below the FP32 normal range 0, above it infinity
__device__ __forceinline__ float
f32_abs(double x)
{
  const uint32_t hi = (uint32_t)__double2hiint(x) & 0x7fffffffu, lo = (uint32_t)__double2loint(x);
  uint32_t       b = (__funnelshift_l(lo, hi, 3) & 0x7fffffffu) ^ 0x40000000u;
  b = hi < 0x38100000u ? 0u : b;
  b = hi >= 0x47f00000u ? 0x7f800000u : b;
  return __uint_as_float(b);
}

__device__ __forceinline__ float
f32_rcp(float x)
{
#ifdef __CUDA_ARCH__
  float r;
  asm("rcp.approx.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
#else
  return host_seed(1.0f / x);
#endif
}
__device__ __forceinline__ float
f32_rsqrt(float x)
{
#ifdef __CUDA_ARCH__
  float r;
  asm("rsqrt.approx.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
#else
  return host_seed(1.0f / sqrtf(x));
#endif
}

// x in FP32, truncated as f32_abs
__device__ __forceinline__ float
f32_of(double x)
{
  return __uint_as_float(__float_as_uint(f32_abs(x)) | ((uint32_t)__double2hiint(x) & 0x80000000u));
}

// Which of several nearly equal speeds is the largest is decided on differences: the FP64 differences of the states'
// values (exact, or nearly) go into FP32. The errors below are relative ones in units of u = 2^-24, to first order:
//   a value or difference cut to FP32 2, a reciprocal of one 4, a reciprocal square root 3 (the approximations are within 2);
//   C, X, Y, Z 10 each; h and m of a state 13 of m (h is a difference of terms as large as m); a difference dC .. dZ 19 of the
//   magnitudes wC .. wZ that it is made of, dm and dh 22 of W / 2.
// The squared speeds are m + s, s = sqrt(disc), so the difference of two is dm + r N with r = 1 / (s0 + sk) and
// N = (h0 + hk) dh + Ck (dY + dZ) + T0 dC. N is off by 28 W (m0 + mk) + 33 W (Ck + T0) at most, of which both factors are
// kept (`e`; with the rest of the sum, and what r adds apart from the next term, 53: kTol is 67). r is off by the error of s:
// disc's is 26 |h| m + 24 disc, so that s's is 13 q + 15, q = |h| m / disc. Next to equal sound and Alfven speeds q is in the
// hundreds, and it multiplies the whole of r N (kRel, 20 with 13 needed). kFloor covers the rounding of the FP64 values
// themselves (within 1e-13 of m where disc is at least 1e-5 m^2) and what FP32 cuts off: a difference of densities, pressures
// or fields below 2^-126 = 1.2e-38 counts as zero, which shifts dm + r N by up to 1000 times its share of d or of d m. With both
// at least 1e-20 that is 2e-15 of m; the upper limits keep the products finite.
constexpr float kTol = 4e-6f, kRel = 1.2e-6f, kFloor = 1e-12f;

// Squared fast speeds along two axes of a state: |b|^2/d and c^2 in FP32 (the field's squares divided by d: X and Y
// along the two axes, Z the third), the square roots of the two discriminants, written as
// ((|b|^2/d - c^2)/2)^2 + c^2 b_t^2/d, free of cancellation, and q (see above).
struct FastEst
{
  float id, C, X, Y, Z, h, m, sx, sy, qx, qy;
};
__device__ __forceinline__ bool
fast_est(float d, float p, float a, float b, float c, float gamma, FastEst & e)
{
  e.id = f32_rcp(d);
  e.C = gamma * p * e.id;
  e.X = a * a * e.id;
  e.Y = b * b * e.id;
  e.Z = c * c * e.id;
  const float t = e.X + e.Y + e.Z;
  e.h = 0.5f * (t - e.C);
  e.m = 0.5f * (t + e.C);
  const float dx = e.h * e.h + e.C * (e.Y + e.Z), dy = e.h * e.h + e.C * (e.X + e.Z);
  const float ix = f32_rsqrt(dx), iy = f32_rsqrt(dy), hm = fabsf(e.h) * e.m;
  e.sx = dx * ix;
  e.sy = dy * iy;
  e.qx = hm * ix * ix;
  e.qy = hm * iy * iy;
  const float least = 1e-5f * e.m * e.m, dm = d * e.m;
  return e.m > 1e-12f && e.m < 1e12f && d > 1e-20f && d < 1e30f && dm > 1e-20f && dm < 1e30f && dx > least && dy > least;
}
// Squared fast speeds of state k less those of state 0 and the bounds of their errors (but for the FP64 values' own). dd, dp,
// da, db, dc: the differences of density, pressure and field; a, b, c: the field's values of the two states.
struct FastDiff
{
  float fx, fy, ex, ey;
};
__device__ __forceinline__ FastDiff
fast_diff(const FastEst & o, const FastEst & k, float dd, float dp, float da, float db, float dc, float a0, float ak,
          float b0, float bk, float c0, float ck, float gamma)
{
  const float ad = fabsf(dd);
  // C, X, Y, Z are quotients by d: the difference is (difference of numerators - quotient of state 0 times dd) / d
  const float dC = k.id * (gamma * dp - o.C * dd), wC = k.id * (gamma * fabsf(dp) + o.C * ad);
  const float dX = k.id * (da * (a0 + ak) - o.X * dd), wX = k.id * (fabsf(da) * (fabsf(a0) + fabsf(ak)) + o.X * ad);
  const float dY = k.id * (db * (b0 + bk) - o.Y * dd), wY = k.id * (fabsf(db) * (fabsf(b0) + fabsf(bk)) + o.Y * ad);
  const float dZ = k.id * (dc * (c0 + ck) - o.Z * dd), wZ = k.id * (fabsf(dc) * (fabsf(c0) + fabsf(ck)) + o.Z * ad);
  const float W = kTol * (wC + wX + wY + wZ);
  const float dt = dX + dY + dZ;
  const float dm = 0.5f * (dt + dC), dh = 0.5f * (dt - dC);
  const float hh = o.h + k.h, mm = o.m + k.m + k.C;
  const float rx = f32_rcp(o.sx + k.sx), ry = f32_rcp(o.sy + k.sy);
  const float Tx = o.Y + o.Z, Ty = o.X + o.Z;
  const float px = rx * (hh * dh + k.C * (dY + dZ) + Tx * dC);
  const float py = ry * (hh * dh + k.C * (dX + dZ) + Ty * dC);
  FastDiff    r;
  r.fx = dm + px;
  r.fy = dm + py;
  r.ex = W * (1.0f + rx * (mm + Tx)) + kRel * (o.qx + k.qx) * fabsf(px);
  r.ey = W * (1.0f + ry * (mm + Ty)) + kRel * (o.qy + k.qy) * fabsf(py);
  return r;
}

// find_speed_fast (models/mhd_utils.h:93-122) of density d, pressure p, squared field b2 and normal field bn
__device__ __forceinline__ double
fast_fp64(double d, double p, double b2, double bn, double gamma)
{
  const Rcp64  id = rcp64(d);
  const double c2 = div64(gamma * p, id);
  const double d2 = dscale_down(div64(b2, id) + c2, 1);
  return sqrt64(d2 + sqrt64(d2 * d2 - div64(c2 * bn * bn, id)));
}

__device__ __forceinline__ bool
dneg(double x)
{
  return __double2hiint(x) < 0;
}

// riemann_hlld (models/RiemannSolvers_MHD.h:311-551); entho = 1 / (gamma - 1)
__device__ __forceinline__ void
riemann_hlld_fp64(double * qL, double * qR, double * flux, double gamma, double entho)
{
  const double a = dscale_down(qL[5] + qR[5], 1);
  const bool   flip = __double_as_longlong(a) < 0 && __double_as_longlong(a) << 1 != 0; // a < 0
  qL[5] = a;
  qR[5] = a;
  const double rl = qL[0], pl = qL[1], ul = qL[2], vl = qL[3], wl = qL[4], bl = qL[6], cl = qL[7];
  const double rr = qR[0], pr = qR[1], ur = qR[2], vr = qR[3], wr = qR[4], br = qR[6], cr = qR[7];
  const double aa = a * a;
  const double b2l = aa + bl * bl + cl * cl, b2r = aa + br * br + cr * cr;
  const double etotl = fma(0.5, b2l, fma(0.5, (ul * ul + vl * vl + wl * wl) * rl, pl * entho));
  const double ptotl = fma(0.5, b2l, pl);
  const double vdotbl = ul * a + vl * bl + wl * cl;
  const double etotr = fma(0.5, b2r, fma(0.5, (ur * ur + vr * vr + wr * wr) * rr, pr * entho));
  const double ptotr = fma(0.5, b2r, pr);
  const double vdotbr = ur * a + vr * br + wr * cr;

  // max(cfastl, cfastr): both only where the estimates do not order them
  double cmax;
  {
    const float fa = f32_abs(a), fbl = f32_of(bl), fcl = f32_of(cl), fbr = f32_of(br), fcr = f32_of(cr);
    const float gf = f32_abs(gamma);
    FastEst     el, er;
    const bool  okl = fast_est(f32_abs(rl), f32_abs(pl), fa, fbl, fcl, gf, el);
    const bool  okr = fast_est(f32_abs(rr), f32_abs(pr), fa, fbr, fcr, gf, er);
    bool        left = true, right = true;
    if (okl && okr && !(dneg(rl) || dneg(rr) || dneg(pl) || dneg(pr)))
    {
      const FastDiff f =
        fast_diff(el, er, f32_of(rr - rl), f32_of(pr - pl), 0.0f, f32_of(br - bl), f32_of(cr - cl), fa, fa, fbl, fbr, fcl, fcr, gf);
      const float tol = f.ex + kFloor * (el.m + er.m);
      left = f.fx <= tol;
      right = f.fx >= -tol;
      // the same state on both sides
      if (left && right && __double_as_longlong(rl) == __double_as_longlong(rr) &&
          __double_as_longlong(pl) == __double_as_longlong(pr) && __double_as_longlong(b2l) == __double_as_longlong(b2r))
        right = false;
    }
    cmax = fast_fp64(left ? rl : rr, left ? pl : pr, left ? b2l : b2r, a, gamma);
    if (left && right)
      cmax = dmax(cmax, fast_fp64(rr, pr, b2r, a, gamma));
  }
  const double sl = dmin(ul, ur) - cmax;
  const double sr = dmax(ul, ur) + cmax;
  const double ml = sl - ul, mr = sr - ur;
  const double rcl = rl * -ml, rcr = rr * mr;
  const Rcp64  irc = rcp64(rcr + rcl);
  const double ustar = div64(rcr * ur + rcl * ul + (ptotl - ptotr), irc);
  const double ptotstar = div64(rcr * ptotl + rcl * ptotr + rcl * rcr * (ul - ur), irc);
  const double pu = ptotstar * ustar, au = ustar * a;

  // star states: side 0 (left), 1 (right)
  double rs[2], vs[2], ws[2], bs[2], cs[2], vb[2], es[2], q[2], sa[2];
#pragma unroll
  for (int k = 0; k < 2; ++k)
  {
    const double r = k ? rr : rl, u = k ? ur : ul, v = k ? vr : vl, w = k ? wr : wl, b = k ? br : bl, c = k ? cr : cl;
    const double m = k ? mr : ml, n = (k ? sr : sl) - ustar;
    const Rcp64  in = rcp64(n);
    const double rm = r * m;
    rs[k] = div64(rm, in);
    const double estar = rm * n - aa;
    const double e = rm * m - aa;
    if (dgt(1e-4 * aa, fabs(estar)))
    {
      vs[k] = v;
      bs[k] = b;
      ws[k] = w;
      cs[k] = c;
    }
    else
    {
      const Rcp64  ie = rcp64(estar);
      const double du = ustar - u;
      vs[k] = v - div64(a * b * du, ie);
      bs[k] = div64(b * e, ie);
      ws[k] = w - div64(a * c * du, ie);
      cs[k] = div64(c * e, ie);
    }
    vb[k] = au + vs[k] * bs[k] + ws[k] * cs[k];
    es[k] = div64(m * (k ? etotr : etotl) - (k ? ptotr : ptotl) * u + pu + a * ((k ? vdotbr : vdotbl) - vb[k]), in);
    q[k] = sqrt64(rs[k]);
    const double ca = div64(fabs(a), rcp64(q[k]));
    sa[k] = k ? ustar + ca : ustar - ca;
  }
  const Rcp64  iq = rcp64(q[0] + q[1]);
  auto         sg = [&](double x) { return flip ? -x : x; }; // times the sign of a
  const double vss = div64(q[0] * vs[0] + q[1] * vs[1] + sg(bs[1] - bs[0]), iq);
  const double wss = div64(q[0] * ws[0] + q[1] * ws[1] + sg(cs[1] - cs[0]), iq);
  const double qq = sg(q[0] * q[1]);
  const double bss = div64(q[0] * bs[1] + q[1] * bs[0] + qq * (vs[1] - vs[0]), iq);
  const double css = div64(q[0] * cs[1] + q[1] * cs[0] + qq * (ws[1] - ws[0]), iq);
  const double vbss = au + vss * bss + wss * css;

  double ro, uo, vo, wo, bo, co, po, eo, vbo;
  if (dpos(sl))
  {
    ro = rl; uo = ul; vo = vl; wo = wl; bo = bl; co = cl;
    po = ptotl; eo = etotl; vbo = vdotbl;
  }
  else if (dpos(sa[0]))
  {
    ro = rs[0]; uo = ustar; vo = vs[0]; wo = ws[0]; bo = bs[0]; co = cs[0];
    po = ptotstar; eo = es[0]; vbo = vb[0];
  }
  else if (dpos(sa[1]))
  {
    const int    k = dpos(ustar) ? 0 : 1;
    const double t = sg(k ? q[1] : q[0]) * ((k ? vb[1] : vb[0]) - vbss);
    ro = k ? rs[1] : rs[0]; uo = ustar; vo = vss; wo = wss; bo = bss; co = css;
    po = ptotstar; eo = k ? es[1] + t : es[0] - t; vbo = vbss;
  }
  else if (dpos(ustar))
  {
    // (ustar > 0 is tested before sar > 0)
    ro = rs[0]; uo = ustar; vo = vss; wo = wss; bo = bss; co = css;
    po = ptotstar; eo = es[0] - sg(q[0]) * (vb[0] - vbss); vbo = vbss;
  }
  else if (dpos(sr))
  {
    ro = rs[1]; uo = ustar; vo = vs[1]; wo = ws[1]; bo = bs[1]; co = cs[1];
    po = ptotstar; eo = es[1]; vbo = vb[1];
  }
  else
  {
    ro = rr; uo = ur; vo = vr; wo = wr; bo = br; co = cr;
    po = ptotr; eo = etotr; vbo = vdotbr;
  }
  const double ru = ro * uo;
  flux[0] = ru;
  flux[1] = (eo + po) * uo - a * vbo;
  flux[2] = ru * uo - aa + po;
  flux[3] = ru * vo - a * bo;
  flux[4] = ru * wo - a * co;
  flux[5] = 0.0;
  flux[6] = bo * uo - a * vo;
  flux[7] = co * uo - a * wo;
}

__device__ __forceinline__ double
sel4(const double * x, int k)
{
  const double lo = k & 1 ? x[1] : x[0], hi = k & 1 ? x[3] : x[2];
  return k & 2 ? hi : lo;
}

__device__ __forceinline__ int
low_bit(uint32_t m)
{
#ifdef __CUDA_ARCH__
  return __ffs((int)m) - 1;
#else
  return __builtin_ctz(m);
#endif
}

// bit k where x[k] (within tol[k]) can be the largest of four
__device__ __forceinline__ uint32_t
screen4(const float * x, const float * tol)
{
  const float t = fmaxf(fmaxf(x[0] - tol[0], x[1] - tol[1]), fmaxf(x[2] - tol[2], x[3] - tol[3]));
  return (x[0] + tol[0] >= t ? 1u : 0u) | (x[1] + tol[1] >= t ? 2u : 0u) | (x[2] + tol[2] >= t ? 4u : 0u) |
         (x[3] + tol[3] >= t ? 8u : 0u);
}

// compute_emf + mag_riemann2d_hlld (models/RiemannSolvers_MHD.h:629-869, 890-1097). The four states around the edge in
// the order LL, LR, RL, RR: density, pressure, velocities u, v and orthogonal field c; the field's transverse
// components are shared, a0 by LL and RL, a1 by LR and RR; b0 by LL and LR, b1 by RL and RR.
__device__ __forceinline__ double
edge_emf_fp64(const double * r, const double * p, const double * u, const double * v, const double * c, double a0,
              double a1, double b0, double b1, double gamma, double smallc)
{
  auto ak = [&](int k) { return k & 1 ? a1 : a0; };
  auto bk = [&](int k) { return k & 2 ? b1 : b0; };
  double b2[4], pt[4];
  {
    const double a00 = a0 * a0, a11 = a1 * a1, b00 = b0 * b0, b11 = b1 * b1;
#pragma unroll
    for (int k = 0; k < 4; ++k)
    {
      b2[k] = ((k & 1 ? a11 : a00) + (k & 2 ? b11 : b00)) + c[k] * c[k];
      pt[k] = fma(0.5, b2[k], p[k]);
    }
  }
  // which of the eight fast speeds can be the largest along their axis
  const float fa0 = f32_of(a0), fa1 = f32_of(a1), fb0 = f32_of(b0), fb1 = f32_of(b1);
  const float fda = f32_of(a1 - a0), fdb = f32_of(b1 - b0);
  float       rf[4];
  double      cmax[2];
  {
    const float gf = f32_abs(gamma);
    uint32_t    mask[2] = {15u, 15u};
    float       fx[4], fy[4], tx[4], ty[4], cf[4];
    FastEst     o;
    bool        ok = !(dneg(r[0]) || dneg(p[0]));
    cf[0] = f32_of(c[0]);
    rf[0] = f32_abs(r[0]);
    ok = fast_est(rf[0], f32_abs(p[0]), fa0, fb0, cf[0], gf, o) && ok;
    fx[0] = fy[0] = 0.0f;
    tx[0] = ty[0] = kFloor * o.m;
#pragma unroll
    for (int k = 1; k < 4; ++k)
    {
      const float ak_f = k & 1 ? fa1 : fa0, bk_f = k & 2 ? fb1 : fb0;
      FastEst     e;
      cf[k] = f32_of(c[k]);
      rf[k] = f32_abs(r[k]);
      ok = ok && !(dneg(r[k]) || dneg(p[k]));
      ok = fast_est(rf[k], f32_abs(p[k]), ak_f, bk_f, cf[k], gf, e) && ok;
      const FastDiff f = fast_diff(o, e, f32_of(r[k] - r[0]), f32_of(p[k] - p[0]), k & 1 ? fda : 0.0f, k & 2 ? fdb : 0.0f,
                                   f32_of(c[k] - c[0]), fa0, ak_f, fb0, bk_f, cf[0], cf[k], gf);
      fx[k] = f.fx;
      fy[k] = f.fy;
      tx[k] = f.ex + kFloor * e.m;
      ty[k] = f.ey + kFloor * e.m;
    }
    if (ok)
    {
      mask[0] = screen4(fx, tx);
      mask[1] = screen4(fy, ty);
      // of two equal states (a region uniform along an axis) only the first
      auto eq = [&](int i, int j) {
        return __double_as_longlong(r[i]) == __double_as_longlong(r[j]) && __double_as_longlong(p[i]) == __double_as_longlong(p[j]) &&
               __double_as_longlong(c[i]) == __double_as_longlong(c[j]);
      };
      const bool ea = __double_as_longlong(a0) == __double_as_longlong(a1), eb = __double_as_longlong(b0) == __double_as_longlong(b1);
      const bool e10 = ea && eq(1, 0), e32 = ea && eq(3, 2), e20 = eb && eq(2, 0), e31 = eb && eq(3, 1);
#pragma unroll
      for (int d = 0; d < 2; ++d)
      {
        uint32_t m = mask[d];
        m = e31 && (m & 2u) ? m & ~8u : m;
        m = e32 && (m & 4u) ? m & ~8u : m;
        m = e20 && (m & 1u) ? m & ~4u : m;
        m = e10 && (m & 1u) ? m & ~2u : m;
        mask[d] = m;
      }
    }
    // the candidates in the scheme's order, each axis's largest kept as it keeps it (r = x > r ? x : r)
    uint32_t todo = mask[0] | (mask[1] << 4);
    cmax[0] = cmax[1] = 0.0;
    uint32_t begun = 0u;
#pragma unroll 1
    while (todo)
    {
      const int j = low_bit(todo);
      todo &= todo - 1u;
      const int    k = j & 3;
      const bool   y = j > 3;
      const double x = fast_fp64(sel4(r, k), sel4(p, k), sel4(b2, k), y ? bk(k) : ak(k), gamma);
      const double old = y ? cmax[1] : cmax[0];
      const bool   take = !(begun & (y ? 2u : 1u)) || dgt(x, old);
      begun |= y ? 2u : 1u;
      if (take)
      {
        if (y)
          cmax[1] = x;
        else
          cmax[0] = x;
      }
    }
  }
  auto most = [&](const double * x) {
    double m = x[0];
    m = dgt(x[1], m) ? x[1] : m;
    m = dgt(x[2], m) ? x[2] : m;
    return dgt(x[3], m) ? x[3] : m;
  };
  auto least = [&](const double * x) {
    double m = x[0];
    m = dgt(m, x[1]) ? x[1] : m;
    m = dgt(m, x[2]) ? x[2] : m;
    return dgt(m, x[3]) ? x[3] : m;
  };
  // (the scheme's order of min/max over the states is LL, LR, RL, RR)
  const double SL = least(u) - cmax[0], SR = most(u) + cmax[0], SB = least(v) - cmax[1], ST = most(v) + cmax[1];
  double       xu[4], yv[4], nx[4], ny[4]; // X - u, Y - v and their products with the density
#pragma unroll
  for (int k = 0; k < 4; ++k)
  {
    xu[k] = (k & 2 ? SR : SL) - u[k];
    yv[k] = (k & 1 ? ST : SB) - v[k];
    nx[k] = r[k] * xu[k];
    ny[k] = r[k] * yv[k];
  }
  // rcLLx = r (u - SL) = -nx and so on for the left and bottom states
  const double ustar = div64(((-nx[0] * u[0] - nx[1] * u[1]) + nx[2] * u[2] + nx[3] * u[3]) + (((pt[0] - pt[2]) + pt[1]) - pt[3]),
                             (nx[2] - (nx[0] + nx[1])) + nx[3]);
  const double vstar = div64(((-ny[0] * v[0] + ny[1] * v[1]) - ny[2] * v[2] + ny[3] * v[3]) + (((pt[0] - pt[1]) + pt[2]) - pt[3]),
                             ((ny[1] - ny[0]) - ny[2]) + ny[3]);
  const double dL = SL - ustar, dR = SR - ustar, dB = SB - vstar, dT = ST - vstar;
  const Rcp64  iL = rcp64(dL), iR = rcp64(dR), iB = rcp64(dB), iT = rcp64(dT);
  double       As[4], Bs[4];
#pragma unroll
  for (int k = 0; k < 4; ++k)
  {
    Bs[k] = div64(bk(k) * xu[k], k & 2 ? iR : iL);
    As[k] = div64(ak(k) * yv[k], k & 1 ? iT : iB);
  }
  // Alfven speeds of the four sides: the largest of |a| / sqrt(rho*x), |A*| / sqrt(rho*) of its two states and smallc.
  // Up to a factor common to the side their squares are v = a^2 / |n| and v (1 + w), n = rho (X - u) and
  // w = ((Y - v) - (Y - v*)) / (Y - v*); bottom and top with x and y exchanged.
  double calf[4];
  {
    float va[4], vb[4], wx[4], wy[4]; // a^2 / |nx|, b^2 / |ny|, v times w
    bool  ok;
    {
      const float fL = f32_rcp(f32_of(dL)), fR = f32_rcp(f32_of(dR)), fB = f32_rcp(f32_of(dB)), fT = f32_rcp(f32_of(dT));
      // a difference cut to zero below 1.2e-38 is then below 1e-14 of dL .. dT
      auto held = [](float x) { return fabsf(x) > 1e-24f && fabsf(x) < 1e24f; };
      ok = held(fL) && held(fR) && held(fB) && held(fT);
#pragma unroll
      for (int k = 0; k < 4; ++k)
      {
        const float gx = f32_of(xu[k] - (k & 2 ? dR : dL)) * (k & 2 ? fR : fL);
        const float gy = f32_of(yv[k] - (k & 1 ? dT : dB)) * (k & 1 ? fT : fB);
        const float fk = k & 1 ? fa1 : fa0, gk = k & 2 ? fb1 : fb0;
        const float nxf = f32_abs(nx[k]), nyf = f32_abs(ny[k]);
        va[k] = fk * fk * f32_rcp(nxf);
        vb[k] = gk * gk * f32_rcp(nyf);
        wx[k] = vb[k] * gx;
        wy[k] = va[k] * gy;
        ok = ok && !dneg(r[k]) && dneg(xu[k]) == dneg(k & 2 ? dR : dL) && dneg(yv[k]) == dneg(k & 1 ? dT : dB);
        ok = ok && nxf > 1e-12f && nxf < 1e12f && nyf > 1e-12f && nyf < 1e12f;
        ok = ok && fabsf(gx) < 1e4f && fabsf(gy) < 1e4f && va[k] < 1e20f && vb[k] < 1e20f;
      }
    }
    const bool za = ok && ((__double_as_longlong(a0) | __double_as_longlong(a1)) << 1) == 0;
    const bool zb = ok && ((__double_as_longlong(b0) | __double_as_longlong(b1)) << 1) == 0;
    // differences of the two states' v along a side: (|n| of the second less |n| of the first)
    const float dnL = -f32_of(nx[0] - nx[1]), dnR = f32_of(nx[2] - nx[3]), dnB = -f32_of(ny[2] - ny[0]), dnT = f32_of(ny[3] - ny[1]);
#pragma unroll 1
    for (int s = 0; s < 4; ++s) // left, right, bottom, top
    {
      // first and second state of the side: LR LL | RR RL | LL RL | LR RR
      const int  k0 = s == 0 ? 1 : (s == 1 ? 3 : (s == 2 ? 0 : 1)), k1 = s == 0 ? 0 : (s == 1 ? 2 : (s == 2 ? 2 : 3));
      const bool y = s >= 2;
      uint32_t   todo = 15u;
      double     m = 0.0;
      bool       begun = false;
      if (y ? zb : za)
      {
        todo = 0u;
        begun = true;
      }
      else if (ok)
      {
        const float v0 = s == 0 ? va[1] : (s == 1 ? va[3] : (s == 2 ? vb[0] : vb[1]));
        const float v1 = s == 0 ? va[0] : (s == 1 ? va[2] : (s == 2 ? vb[2] : vb[3]));
        const float w0 = s == 0 ? wy[1] : (s == 1 ? wy[3] : (s == 2 ? wx[0] : wx[1]));
        const float w1 = s == 0 ? wy[0] : (s == 1 ? wy[2] : (s == 2 ? wx[2] : wx[3]));
        const float dn = s == 0 ? dnL : (s == 1 ? dnR : (s == 2 ? dnB : dnT));
        // second less first: ((f1 - f0)(f1 + f0) - v0 dn) / |n1|
        const float df = y ? fdb : -fda, f0 = y ? fb0 : fa1, f1 = y ? fb1 : fa0;
        const float in = f32_rcp(s == 0 ? f32_abs(nx[0]) : (s == 1 ? f32_abs(nx[2]) : (s == 2 ? f32_abs(ny[2]) : f32_abs(ny[3]))));
        const float dv = in * (df * (f0 + f1) - v0 * dn), ev = in * (fabsf(df) * (fabsf(f0) + fabsf(f1)) + v0 * fabsf(dn));
        const float fl = kFloor * fmaxf(v0, v1);
        const float e[4] = {0.0f, w0, dv, dv + w1};
        const float t[4] = {fl, kTol * fabsf(w0) + fl, kTol * ev + fl, kTol * (ev + fabsf(w1)) + fl};
        todo = screen4(e, t);
        // (products of the fields are off by up to 1e-45 below 1e-38: less than kFloor of a square of 1e-32)
        todo = fmaxf(v0, v1) > 1e-25f && fmaxf(fabsf(f0), fabsf(f1)) > 1e-16f ? todo : 15u;
      }
      // num / sqrt(rho) grows with num and falls with rho, rounded as well: of two candidates ordered in both only one
      // is evaluated (a uniform state's four differ by roundings of rho and num, if at all)
      double num = 0.0, rho = 0.0;
      bool   held = false;
#pragma unroll 1
      while (true)
      {
        const bool have = todo != 0u;
        double     num1 = 0.0, rho1 = 0.0;
        if (have)
        {
          const int j = low_bit(todo);
          todo &= todo - 1u;
          const int    k = j & 2 ? k1 : k0;
          const bool   star = j & 1;
          const bool   byx = star || !y; // rho* of a side along x, or of the corner, starts from the x wave
          const Rcp64  ix = k & 2 ? iR : iL, iy = k & 1 ? iT : iB;
          const double nxk = sel4(nx, k), nyk = sel4(ny, k);
          Rcp64        i0;
          i0.y = byx ? ix.y : iy.y;
          i0.R = byx ? ix.R : iy.R;
          rho1 = div64(byx ? nxk : nyk, i0);
          if (star)
            rho1 = div64(rho1 * sel4(yv, k), iy);
          num1 = fabs(star ? (y ? sel4(Bs, k) : sel4(As, k)) : (y ? bk(k) : ak(k)));
        }
        // (ok: both are non-negative numbers, whose bit patterns are in their order)
        const int64_t dn = (int64_t)(__double_as_longlong(num1) - __double_as_longlong(num)),
                      dr = (int64_t)(__double_as_longlong(rho1) - __double_as_longlong(rho));
        const bool below = ok && dn <= 0 && dr >= 0, above = ok && dn >= 0 && dr <= 0;
        if (held && !(have && (below || above)))
        {
          const double x = div64(num, rcp64(sqrt64(rho)));
          if (!begun || dgt(x, m))
            m = x;
          begun = true;
        }
        if (!have)
          break;
        if (!held || !below)
        {
          num = num1;
          rho = rho1;
        }
        held = true;
      }
      m = dgt(smallc, m) ? smallc : m;
      if (s == 0)
        calf[0] = m;
      else if (s == 1)
        calf[1] = m;
      else if (s == 2)
        calf[2] = m;
      else
        calf[3] = m;
    }
  }
  const double SAL = dmin(ustar - calf[0], 0.0), SAR = dmax(ustar + calf[1], 0.0);
  const double SAB = dmin(vstar - calf[2], 0.0), SAT = dmax(vstar + calf[3], 0.0);
  const Rcp64  iRL = rcp64(SAR - SAL), iTB = rcp64(SAT - SAB);
  const bool   sbn = dneg(SB), stn = dneg(ST), sln = dneg(SL), srn = dneg(SR);
  if (sbn && !stn && sln && !srn)
  {
    double E[4];
#pragma unroll
    for (int k = 0; k < 4; ++k)
      E[k] = ustar * Bs[k] - vstar * As[k];
    const double AT = div64(SAR * As[3] - SAL * As[1], iRL), AB = div64(SAR * As[2] - SAL * As[0], iRL);
    const double BR = div64(SAT * Bs[3] - SAB * Bs[2], iTB), BL = div64(SAT * Bs[1] - SAB * Bs[0], iTB);
    return div64(div64(SAL * SAB * E[3] - SAL * SAT * E[2] - SAR * SAB * E[1] + SAR * SAT * E[0], iRL), iTB) -
           div64(SAT * SAB, iTB) * (AT - AB) + div64(SAR * SAL, iRL) * (BR - BL);
  }
  // the scheme's sum over all regions, with weights 0 and 1, is NaN where any wave speed or star field is not finite
  bool bad = false;
#pragma unroll
  for (int k = 0; k < 4; ++k)
    bad = bad || dspecial(As[k]) || dspecial(Bs[k]);
  if (bad || dspecial(SL) || dspecial(SR) || dspecial(SB) || dspecial(ST) || dspecial(SAL) || dspecial(SAR) || dspecial(SAB) ||
      dspecial(SAT) || dspecial(ustar) || dspecial(vstar))
    return __longlong_as_double(0x7ff8000000000000ll);
  // the wave fan lies on one side of the edge along an axis (or both): k0, k1 the two states of that side
  if (!sbn || stn)
  {
    const int k0 = sbn ? 1 : 0, k1 = k0 + 2; // bottom: LL, RL; top: LR, RR
    if (!sln || srn)
    {
      const int k = sln ? k1 : k0;
      return sel4(u, k) * bk(k) - sel4(v, k) * ak(k);
    }
    const double E0 = ustar * sel4(Bs, k0) - sel4(v, k0) * ak(k0), E1 = ustar * sel4(Bs, k1) - sel4(v, k1) * ak(k1);
    return div64(SAR * E0 - SAL * E1 + SAR * SAL * (b1 - b0), iRL);
  }
  const int    k0 = sln ? 2 : 0, k1 = k0 + 1; // left: LL, LR; right: RL, RR
  const double E0 = sel4(u, k0) * bk(k0) - vstar * sel4(As, k0), E1 = sel4(u, k1) * bk(k1) - vstar * sel4(As, k1);
  return div64(SAT * E0 - SAB * E1 - SAT * SAB * (a1 - a0), iTB);
}

} // namespace gmhd
