"""FP64 steps of meshes with few tiles: the smaller default tiles and their wide variants, on both sides of the limits
(half the SMs' worth of tiles), against the oracle bit for bit."""
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
