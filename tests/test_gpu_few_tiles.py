"""Steps of meshes with few tiles: the smaller default tiles and their wide variants, on both sides of the limits (half the
SMs' worth of tiles, two small tiles an SM): FP64 against the oracle bit for bit, mixed against the same cells as a part of
a mesh with many tiles."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from godunov_mhd_ct_gb300 import workloads as wl  # noqa: E402
from godunov_mhd_ct_gb300.mesh import BlockMesh  # noqa: E402
from godunov_mhd_ct_gb300.solver import GodunovImplemGB300  # noqa: E402

from .helpers import oracle_mesh, oracle_settings, settings  # noqa: E402

pytestmark = pytest.mark.gpu


# tiles of the largest kind: 64, 80, 4 (2D 16x16); 32, 80 (3D 8x4x4); 4x4x4 tiles only: 27, 216; 8x8 only: 64, 320
@pytest.mark.parametrize("dim,bricks,level,block", [(2, 1, 3, 16), (2, 5, 2, 16), (2, 1, 1, 16), (3, 1, 1, 8), (3, 1, 0, 16),
                                                    (3, 5, 1, 8), (3, 1, 0, 12), (3, 1, 1, 12), (2, 1, 3, 8), (2, 5, 3, 8)])
def test_few_tiles_fp64(oracle_lib, dim, bricks, level, block):
    mesh = BlockMesh.uniform(dim, bricks=(bricks, 1, 1), level=level, block=(block, block, block if dim == 3 else 1))
    st = settings()
    U, B = wl.random_smooth(mesh, gamma=st.gamma0, seed=block + bricks)
    om, os_ = oracle_mesh(oracle_lib, mesh), oracle_settings(oracle_lib, st)
    dt = st.cfl / oracle_lib.inv_dt(om, os_, U, B)
    U2o, B2o = oracle_lib.step(om, os_, U, B, dt)
    impl = GodunovImplemGB300(st, mesh, precision="fp64")
    dU, dB = torch.from_numpy(U).cuda(), torch.from_numpy(B).cuda()
    dU2, dB2 = torch.zeros_like(dU), torch.zeros_like(dB)
    impl.do_time_step(dU, dU2, dB, dB2, dt)
    assert np.array_equal(dU2.cpu().numpy(), U2o) and np.array_equal(dB2.cpu().numpy(), B2o)
    impl.close()


# a mesh of `bricks` like bricks against one of `many` of them, all alike: the first takes the small tiles, the second the
# large ones, and its first bricks are the same cells with the same neighbours. The rounding of a tile is its kind's, so
# the results are equal.
@pytest.mark.parametrize("dim,level,block,many", [(2, 0, 16, 80), (2, 3, 16, 2), (2, 1, 48, 4), (3, 0, 8, 80), (3, 1, 16, 2),
                                                  (2, 1, 8, 80), (3, 1, 4, 40), (3, 0, 12, 12), (2, 1, 24, 12)])
@pytest.mark.parametrize("riemann", ["HLLD", "LLF"])
def test_few_tiles_mixed(dim, level, block, many, riemann):
    st = settings(riemann=riemann)
    out = []
    for bricks in (1, many):
        mesh = BlockMesh.uniform(dim, bricks=(bricks, 1, 1), level=level, block=(block, block, block if dim == 3 else 1))
        one = BlockMesh.uniform(dim, level=level, block=(block, block, block if dim == 3 else 1))
        U, B = wl.random_smooth(one, gamma=st.gamma0, seed=block)
        at = {tuple(c): n for n, c in enumerate(one.coords[: one.n_owned].tolist())}
        side = 1 << level
        pick = [at[(c[0] % side, c[1] % side, c[2] % side)] for c in mesh.coords[: mesh.n_owned].tolist()]
        dU, dB = torch.from_numpy(U[pick]).cuda(), torch.from_numpy(B[pick]).cuda()
        dU2, dB2 = torch.zeros_like(dU), torch.zeros_like(dB)
        impl = GodunovImplemGB300(st, mesh, precision="mixed")
        impl.do_time_step(dU, dU2, dB, dB2, 0.1 * one.block_dx().min())
        first = {tuple(c): n for n, c in enumerate(mesh.coords[: mesh.n_owned].tolist())}
        sel = [first[tuple(c)] for c in one.coords[: one.n_owned].tolist()]
        out.append((dU2[sel].cpu().numpy(), dB2[sel].cpu().numpy()))
        impl.close()
    assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])
