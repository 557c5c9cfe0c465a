"""The mixed step's default tile on meshes of few tiles against the largest tile asked for by name, and gmhd_step_host, which
always steps in the largest: the same bits with every solver, limiter and source, in smooth and in supersonic flow."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from godunov_mhd_ct_gb300 import workloads as wl  # noqa: E402
from godunov_mhd_ct_gb300.mesh import BlockMesh  # noqa: E402
from godunov_mhd_ct_gb300.solver import GodunovImplemGB300  # noqa: E402

from .helpers import settings  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,level,block,largest", [(2, 3, 16, 16), (2, 2, 16, 16), (3, 2, 8, 8), (3, 1, 16, 8)])
@pytest.mark.parametrize("riemann", ["HLLD", "HLL", "LLF", "HLLC"])
@pytest.mark.parametrize("slope_type", [1.0, 2.0])
@pytest.mark.parametrize("gravity", [False, True])
@pytest.mark.parametrize("speed", [0.0, 4.0])
def test_default_tile_gives_the_largest_tiles_bits(dim, level, block, largest, riemann, slope_type, gravity, speed):
    mesh = BlockMesh.uniform(dim, level=level, block=(block, block, block if dim == 3 else 1))
    st = settings(riemann=riemann, slope_type=slope_type)
    if gravity:
        st.gravity = (0.1, -0.3, 0.2)
    U, B = wl.random_smooth(mesh, gamma=st.gamma0, seed=level)
    n = mesh.n_owned
    for d in range(dim):  # a part of the mesh moves, and every cell a little at random
        kick = speed * (np.arange(n) > n // 3)[:, None, None, None] * (-1.0) ** d
        kick = kick + 0.05 * np.random.default_rng(d).standard_normal(U[:, 0].shape)
        v = U[:, 2 + d] / U[:, 0]
        U[:, 1] += 0.5 * U[:, 0] * ((v + kick) ** 2 - v ** 2)
        U[:, 2 + d] += U[:, 0] * kick
    dt = 0.05 * float(mesh.block_dx().min())
    impl = GodunovImplemGB300(st, mesh, precision="mixed")
    dU, dB = torch.from_numpy(U).cuda(), torch.from_numpy(B).cuda()
    out = []
    for tile in (0, largest):
        impl.set_tile(tile)
        dU2, dB2 = torch.zeros_like(dU), torch.zeros_like(dB)
        impl.do_time_step(dU, dU2, dB, dB2, dt)
        out.append((dU2.cpu().numpy(), dB2.cpu().numpy()))
    impl.set_tile(0)
    out.append(impl.step_host(U, B, dt)[:2])
    impl.close()
    assert np.all(np.isfinite(out[0][0]))
    for U2, B2 in out[1:]:
        assert np.array_equal(out[0][0], U2) and np.array_equal(out[0][1], B2)
