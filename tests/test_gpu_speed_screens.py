"""FP64 steps of states in which the FP32 screens of the exact path are least certain, against the oracle bit for bit, with the
GPU's own approximate reciprocals: sound and Alfven speeds nearly equal, densities down to 1e-30 with floors below them, and
thin gas at rest in fields near the end of the FP32 range."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from godunov_mhd_ct_gb300 import workloads as wl  # noqa: E402
from godunov_mhd_ct_gb300.mesh import BlockMesh  # noqa: E402
from godunov_mhd_ct_gb300.solver import GodunovImplemGB300  # noqa: E402

from .helpers import oracle_mesh, oracle_settings, settings  # noqa: E402

pytestmark = pytest.mark.gpu


def _state(mesh, rho0, v0, field, p0, spread, transverse, seed):
    """Cells within `spread` of one another; a normal field along one axis, transverse fields weaker by `transverse`."""
    U, B = mesh.alloc_state()
    n, dim, axis = mesh.n_owned, mesh.dim, seed % mesh.dim
    g = [a[:n].astype(np.int64) for a in mesh.global_cell_index()]
    rand = lambda s, ids: 2.0 * wl.uniform01(100 * seed + s, ids.astype(np.uint64)) - 1.0
    cell = g[0] + (g[1] << 13) + (g[2] << 26)
    rho = rho0 * (1.0 + spread * rand(0, cell))
    p = p0 * (1.0 + spread * rand(1, cell))
    vel = [v0 * rand(2 + d, cell) for d in range(3)]
    F, bc = mesh.split_faces(B), []
    for d in range(3):  # each component varies along one other axis only
        b = field * (1.0 + spread * rand(5 + d, g[(d + 1) % dim]))
        if d != axis:
            b = b * transverse * (1.0 + 0.3 * rand(8 + d, g[(d + 1) % dim]))
        bc.append(b)
        ax = 3 - d
        F[d][:n] = b if dim == 2 and d == 2 else np.concatenate([b, np.take(b, [0], axis=ax)], axis=ax)
    U[:n, 0] = rho
    for d in range(3):
        U[:n, 2 + d] = rho * vel[d]
    U[:n, 1] = p / 0.4 + 0.5 * rho * (vel[0] ** 2 + vel[1] ** 2 + vel[2] ** 2) + 0.5 * (bc[0] ** 2 + bc[1] ** 2 + bc[2] ** 2)
    return U, B


@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("kind", ["degenerate", "thin", "weak"])
@pytest.mark.parametrize("seed", range(6))
def test_step_equals_the_oracle(oracle_lib, dim, kind, seed):
    mesh = BlockMesh.uniform(dim, level=2 if dim == 2 else 1, block=(16, 16, 16 if dim == 3 else 1))
    rng = np.random.default_rng(seed)
    st = settings(gamma0=1.4, cfl=0.4)
    spread = 10.0 ** rng.uniform(-10, -3)
    if kind == "degenerate":  # p = B^2 / gamma: sound speed = Alfven speed, or close to it
        near = 0.0 if seed % 2 else 10.0 ** rng.uniform(-3.5, -1.5)
        U, B = _state(mesh, 1.0, 0.3, 1.0, (1.0 + near) / 1.4, spread, 10.0 ** rng.uniform(-4, -1), seed)
    else:
        st.smallr = st.smallc = 1e-40
        rho0, v0 = 10.0 ** rng.uniform(-30, -24) if kind == "thin" else 10.0 ** rng.uniform(-12, -10), 10.0 ** rng.uniform(-4, 1)
        field = np.sqrt(rho0) * v0 if kind == "thin" else 10.0 ** rng.uniform(-17.5, -16)
        U, B = _state(mesh, rho0, 0.3 * v0 if kind == "thin" else 0.0, field, rho0 * v0 * v0, spread, 0.3, seed)
    om, os_ = oracle_mesh(oracle_lib, mesh), oracle_settings(oracle_lib, st)
    inv = oracle_lib.inv_dt(om, os_, U, B)
    U2o, B2o = oracle_lib.step(om, os_, U, B, st.cfl / inv)
    impl = GodunovImplemGB300(st, mesh, precision="fp64")
    dU, dB = torch.from_numpy(U).cuda(), torch.from_numpy(B).cuda()
    dU2, dB2 = torch.zeros_like(dU), torch.zeros_like(dB)
    assert impl.compute_inv_dt(dU, dB) == inv
    impl.do_time_step(dU, dU2, dB, dB2, st.cfl / inv)
    impl.close()
    assert np.all(np.isfinite(U2o))
    assert np.array_equal(dU2.cpu().numpy(), U2o) and np.array_equal(dB2.cpu().numpy(), B2o)
