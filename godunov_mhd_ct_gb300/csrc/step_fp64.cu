// FP64 instantiations of the fused step: the drop-in path. This unit is compiled with
// --fmad=false so that every a*b+c stays unfused, matching the reference formulas' FP64 rounding.
#include <type_traits>

#include "cfl_screen.cuh"
#include "launch.cuh"

namespace gmhd
{
// Threads per tile: 128^3 Orszag-Tang took 18.7 / 17.6 / 17.6 ms with 256 / 384 / 512 threads on the 8x4x4 tile
// (one CTA per SM either way, by its shared memory), a blast at rest 21.2 / 20.4 / 18.7 ms; blocks of 12^3 (4x4x4
// tiles) 12.2 ms with 64 threads, 8.2 with 128. The wide variants (_W) are for a launch of so few tiles that each SM
// holds one or two: 2D 128^2 in 8x8 tiles 131 us with 64 threads, 94 with 128; 16^3 cells in 4x4x4 tiles 156 us with
// 128 threads, 119 with 256.
// 8x4x4, one CTA an SM: Orszag-Tang 64^3, ms a step: 2.16 with 384 threads, 2.16 with 512, 1.97 with 576, 2.01 with 640,
// 2.05 with 768; shear layers with coarse/fine faces 18.04, 17.62, 16.25, 16.31, 16.46.
using F64_3D_844 = Cfg<double, 3, 8, 4, 4, 576, true>;
using F64_3D_444 = Cfg<double, 3, 4, 4, 4, 128, true>;
using F64_3D_444_W = Cfg<double, 3, 4, 4, 4, 256, true>;
using F64_2D_16 = Cfg<double, 2, 16, 16, 1, 256, true>;
using F64_2D_8 = Cfg<double, 2, 8, 8, 1, 64, true>;
using F64_2D_8_W = Cfg<double, 2, 8, 8, 1, 128, true>;
using F64_2D_4 = Cfg<double, 2, 4, 4, 1, 32, true>;
using F64_3D_844_AMR = Cfg<double, 3, 8, 4, 4, 576, true, true>;
using F64_3D_444_AMR = Cfg<double, 3, 4, 4, 4, 128, true, true>;
using F64_2D_16_AMR = Cfg<double, 2, 16, 16, 1, 256, true, true>;
using F64_2D_8_AMR = Cfg<double, 2, 8, 8, 1, 64, true, true>;
using F64_2D_4_AMR = Cfg<double, 2, 4, 4, 1, 32, true, true>;

template <bool AMR>
int
launch_step_fp64_cfg(const StepArgs & a, int dim, cudaStream_t stream)
{
  int       cand[3];
  const int x = pick_tile(cand, tile_candidates_fp64(dim, a.bx, a.by, a.bz, false, cand), a.tile);
  const int t = dim == 3 ? 4 : x;
  const long long tiles =
    x <= 0 ? 0 : (a.tile_list ? (long long)a.n_list : (long long)a.n_owned * (a.bx / t) * (a.by / t) * (dim == 3 ? a.bz / t : 1));
  if (dim == 3)
  {
    if (x == 8)
      return launch_fused<std::conditional_t<AMR, F64_3D_844_AMR, F64_3D_844>>(a, stream);
    if (!AMR && tiles <= kSMs)
      return launch_fused<F64_3D_444_W>(a, stream);
    return launch_fused<std::conditional_t<AMR, F64_3D_444_AMR, F64_3D_444>>(a, stream);
  }
  if (x == 16)
    return launch_fused<std::conditional_t<AMR, F64_2D_16_AMR, F64_2D_16>>(a, stream);
  if (x == 8 && !AMR && tiles <= 2 * kSMs)
    return launch_fused<F64_2D_8_W>(a, stream);
  if (x == 8)
    return launch_fused<std::conditional_t<AMR, F64_2D_8_AMR, F64_2D_8>>(a, stream);
  return launch_fused<std::conditional_t<AMR, F64_2D_4_AMR, F64_2D_4>>(a, stream);
}

int
launch_step_fp64(const StepArgs & a, int dim, cudaStream_t stream)
{
  if (a.src.viscosity)
    return launch_step_fp64_visc(a, dim, stream);
  return a.kind ? launch_step_fp64_cfg<true>(a, dim, stream) : launch_step_fp64_cfg<false>(a, dim, stream);
}

int
tile_candidates_fp64(int dim, int bx, int by, int bz, bool /*visc: same tiles*/, int * out)
{
  int n = 0;
  if (dim == 3)
  {
    // 8x4x4 tiles, then 4x4x4
    if (bx % 8 == 0 && by % 4 == 0 && bz % 4 == 0)
      out[n++] = 8;
    if (bx % 4 == 0 && by % 4 == 0 && bz % 4 == 0)
      out[n++] = 4;
    return n;
  }
  for (int t : {16, 8, 4})
    if (bx % t == 0 && by % t == 0)
      out[n++] = t;
  return n;
}

void
tile_shape_fp64(int dim, int bx, int by, int bz, bool visc, int tile, int * t)
{
  int       cand[3];
  const int x = pick_tile(cand, tile_candidates_fp64(dim, bx, by, bz, visc, cand), tile);
  if (dim == 3)
  {
    t[0] = x == 8 ? 8 : 4;
    t[1] = 4;
    t[2] = 4;
    return;
  }
  const int n = x ? x : 4;
  t[0] = t[1] = n;
  t[2] = 1;
}

int
default_tile_fp64(int dim, int bx, int by, int bz, int n_owned)
{
  // (FP64 results do not depend on the tile.) Largest against small tiles, us a step. Uniform, small ones _W: 2D, 64 tiles of
  // 16x16 138 / 81, 80 138 / 130; 3D, 64 tiles of 8x4x4 146 / 107, 96 145 / 175. Without a _W variant the small tiles gain less.
  // Coarse/fine: 2D, 22 to 76 tiles 295 / 250, with viscosity 320 / 266 (88 298 / 261, 323 / 276: the line could lie
  // higher there); 3D, 60 tiles 325 / 319, with viscosity 367 / 358, 116 tiles 326 / 356, 367 / 397. Uniform with viscosity:
  // 2D, 1 to 64 tiles 147 / 120, 80 146 / 135; 3D, 64 tiles 161 / 158, 96 161 / 190.
  const long long half = kSMs / 2;
  if (dim == 2 && bx % 16 == 0 && by % 16 == 0 && (long long)n_owned * (bx / 16) * (by / 16) <= half)
    return 8;
  if (dim == 3 && bx % 8 == 0 && by % 4 == 0 && bz % 4 == 0 && (long long)n_owned * (bx / 8) * (by / 4) * (bz / 4) <= half)
    return 4;
  return 0;
}

int
prepare_fp64()
{
  int rc = 0;
  rc = rc ? rc : prepare_fused<F64_3D_844>();
  rc = rc ? rc : prepare_fused<F64_3D_444>();
  rc = rc ? rc : prepare_fused<F64_3D_444_W>();
  rc = rc ? rc : prepare_fused<F64_2D_8_W>();
  rc = rc ? rc : prepare_fused<F64_2D_16>();
  rc = rc ? rc : prepare_fused<F64_2D_8>();
  rc = rc ? rc : prepare_fused<F64_2D_4>();
  rc = rc ? rc : prepare_fused<F64_3D_844_AMR>();
  rc = rc ? rc : prepare_fused<F64_3D_444_AMR>();
  rc = rc ? rc : prepare_fused<F64_2D_16_AMR>();
  rc = rc ? rc : prepare_fused<F64_2D_8_AMR>();
  rc = rc ? rc : prepare_fused<F64_2D_4_AMR>();
  return rc;
}
} // namespace gmhd

namespace gmhd
{
// ComputeDtMHDFunctor::compute_cfl (scheme/ComputeDtMHDFunctor.cpp:86-151) over the owned blocks, max-reduced
// per problem: FP64 with the reference operand order where the FP32 screen (cfl_screen.cuh) leaves a cell in
// question. A CTA takes 1024 cells of one block, so that a mesh of few large blocks fills the device too: one
// CTA per 32^3 block left 152 SMs with 3.4 CTAs each.
__global__ void __launch_bounds__(256)
inv_dt_kernel(const double * __restrict__ U, const double * __restrict__ B, const int32_t * __restrict__ level,
              const int32_t * __restrict__ problem, int chunks, int dim, int bx, int by, int64_t ncell, int64_t nfx,
              int64_t nfy, int64_t nface, double gamma0, float gm1, double smallr, double smallp,
              double scaling_factor, float inv_scaling, Sources src, unsigned long long * invdt)
{
  const int     blk = blockIdx.x / chunks, chunk = blockIdx.x - blk * chunks;
  const int64_t cells = (int64_t)bx << level[blk];
  auto          dx_of = [&]() { return (1.0 / (double)cells) * scaling_factor; };
  screened_inv_dt(U + (int64_t)blk * 5 * ncell, B + (int64_t)blk * nface, dim, bx, by,
                  (int64_t)chunk * 256 * kScreenCells, ncell, nfx, nfy, (float)cells * inv_scaling, gamma0, gm1, smallr,
                  smallp, src, dx_of, &invdt[problem ? problem[blk] : 0]);
}

int
launch_inv_dt(const double * U, const double * B, const int32_t * level, const int32_t * problem, int n_owned, int dim,
              int bx, int by, int bz, int64_t ncell, int64_t nfx, int64_t nfy, int64_t nface, double gamma0,
              double smallr, double smallp, double scaling_factor, const Sources & src, unsigned long long * invdt,
              cudaStream_t stream)
{
  if (n_owned <= 0)
    return 0;
  (void)bz;
  const int64_t chunks = (ncell + 256 * kScreenCells - 1) / (256 * kScreenCells);
  if (ncell > 0xffffffffLL || (int64_t)n_owned * chunks > 0x7fffffffLL)
    return (int)cudaErrorInvalidConfiguration;
  inv_dt_kernel<<<(unsigned)(n_owned * chunks), 256, 0, stream>>>(U, B, level, problem, (int)chunks, dim, bx, by, ncell,
                                                                  nfx, nfy, nface, gamma0, (float)(gamma0 - 1.0), smallr,
                                                                  smallp, scaling_factor, (float)(1.0 / scaling_factor), src, invdt);
  return (int)cudaGetLastError();
}
} // namespace gmhd
