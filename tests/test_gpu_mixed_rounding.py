"""Every kernel of the mixed step rounds as it always has: SHA-256 digests of one step's U2 and B2, recorded before the edge
solver, HLLD and the gravity kick named their roundings. (The other phases' FP32 contractions are the compiler's: another nvcc may need new
digests.) States come from integer hashes and plain arithmetic only, so that the host's math library has no part in them."""
import hashlib

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from godunov_mhd_ct_gb300 import workloads as wl  # noqa: E402
from godunov_mhd_ct_gb300.mesh import BlockMesh  # noqa: E402
from godunov_mhd_ct_gb300.settings import MHDSettings  # noqa: E402
from godunov_mhd_ct_gb300.solver import GodunovImplemGB300  # noqa: E402

pytestmark = pytest.mark.gpu


def _corner(level, lo, hi):
    return max(lo) < 0.25


def _mesh(dim, block, amr):
    b = (block, block, block if dim == 3 else 1)
    if amr:
        return BlockMesh.amr(dim, _corner, base_level=2 if dim == 2 else 1, max_level=4 if dim == 2 else 2, block=b)
    return BlockMesh.uniform(dim, level=4 if dim == 2 else 2, block=b)


def _state(mesh):
    U, B = mesh.alloc_state()
    n, dim = mesh.n_owned, mesh.dim
    g = [a[:n].astype(np.int64) for a in mesh.global_cell_index()]
    level = mesh.level[:n].astype(np.int64)[:, None, None, None]
    rand = lambda seed, ids: 2.0 * wl.uniform01(seed, ids.astype(np.uint64)) - 1.0
    cell = g[0] + (g[1] << 12) + (g[2] << 24) + (level << 36)
    rho, p = 1.0 + 0.4 * rand(1, cell), 1.0 + 0.4 * rand(2, cell)
    vel = [0.5 * rand(3 + d, cell) for d in range(3)]
    # each component of B varies along one other axis only: divergence-free, equal on both copies of a face
    F = mesh.split_faces(B)
    bc = []
    for d in range(3):
        along = (d + 1) % dim
        b = 0.5 + 0.4 * rand(8 + d, g[along] + (level << 36))
        bc.append(b)
        if dim == 2 and d == 2:
            F[2][:n] = b
        else:
            ax = 3 - d
            F[d][:n] = np.concatenate([b, np.take(b, [0], axis=ax)], axis=ax)
    U[:n, 0] = rho
    for d in range(3):
        U[:n, 2 + d] = rho * vel[d]
    U[:n, 1] = p / 0.4 + 0.5 * rho * (vel[0] ** 2 + vel[1] ** 2 + vel[2] ** 2) + 0.5 * (bc[0] ** 2 + bc[1] ** 2 + bc[2] ** 2)
    return U, B


def digest(dim, block, amr, mu, gravity=None, dt=2.0 ** -13):
    mesh = _mesh(dim, block, amr)
    impl = GodunovImplemGB300(MHDSettings(gamma0=1.4, cfl=0.4, slope_type=2.0, riemann="HLLD", viscosity_mu=mu or None,
                                          gravity=gravity), mesh, precision="mixed")
    U, B = (torch.from_numpy(a).cuda() for a in _state(mesh))
    U2, B2 = torch.zeros_like(U), torch.zeros_like(B)
    impl.do_time_step(U, U2, B, B2, dt)
    n = mesh.n_owned
    out = hashlib.sha256(U2[:n].cpu().numpy().tobytes() + B2[:n].cpu().numpy().tobytes()).hexdigest()[:16]
    impl.close()
    return out


DIGESTS = {
    (2, 16, False, 0.0): "9ff6b74fc4f8935e",
    (2, 16, False, 0.001): "3f5e07d17ee085ca",
    (2, 16, True, 0.0): "dcaf600ba090673c",
    (2, 16, True, 0.001): "822bbad5a1676448",
    (2, 8, False, 0.0): "aae81f8de0653322",
    (2, 8, False, 0.001): "d25ead4f0c455dc9",
    (2, 8, True, 0.0): "f3cef1b233c193a1",
    (2, 8, True, 0.001): "8078de55113896f2",
    (2, 12, False, 0.0): "9111fa114a5a61b6",
    (2, 12, False, 0.001): "866d7fb7b4502de1",
    (2, 12, True, 0.0): "7e9dec5f74513648",
    (2, 12, True, 0.001): "a02aff7032b9a69a",
    (3, 16, False, 0.0): "b4624cf0dad29b6a",
    (3, 16, False, 0.001): "6b4d7df3096dde8d",
    (3, 16, True, 0.0): "fc6a5e82f4f1a094",
    (3, 16, True, 0.001): "78616872ea53dffe",
    (3, 12, False, 0.0): "91ffafe1736d7b0e",
    (3, 12, False, 0.001): "736dd7a5698f4d9f",
    (3, 12, True, 0.0): "1fc4dc76bb130549",
    (3, 12, True, 0.001): "1fabcd6378a51a41",
}


@pytest.mark.parametrize("dim,block", [(2, 16), (2, 8), (2, 12), (3, 16), (3, 12)])
@pytest.mark.parametrize("amr", [False, True])
@pytest.mark.parametrize("mu", [0.0, 1e-3])
def test_step_rounds_as_recorded(dim, block, amr, mu):
    assert digest(dim, block, amr, mu) == DIGESTS[dim, block, amr, mu]


# strong gravity along every axis, a time step that is no power of two (with one, the kick's product is exact)
GRAVITY = dict(gravity=(40.0, -70.0, 55.0), dt=1.1371 * 2.0 ** -13)
DIGESTS_GRAVITY = {
    (2, 16, False, 0.0): "464faf66387fafe9",
    (2, 16, False, 0.001): "355e386b6b450ab5",
    (2, 16, True, 0.0): "7b849d38a8255a06",
    (2, 16, True, 0.001): "079effc793a5bd62",
    (2, 8, False, 0.0): "72e6feceb810ea53",
    (2, 8, False, 0.001): "b22418929c599d21",
    (2, 8, True, 0.0): "007f86afb3612fb7",
    (2, 8, True, 0.001): "206cc47310802d64",
    (2, 12, False, 0.0): "7d1e60551e9d7839",
    (2, 12, False, 0.001): "22bfba4ceaf106b1",
    (2, 12, True, 0.0): "7ea97a9095eab997",
    (2, 12, True, 0.001): "3b050312b9a4573e",
    (3, 16, False, 0.0): "b865db712fa14198",
    (3, 16, False, 0.001): "5d408451215c48a7",
    (3, 16, True, 0.0): "e4a137b032fbf704",
    (3, 16, True, 0.001): "e5dcca840486961f",
    (3, 12, False, 0.0): "c4a6917d8e3265f5",
    (3, 12, False, 0.001): "d30e02fa96c80de9",
    (3, 12, True, 0.0): "b722a3a2d1896a62",
    (3, 12, True, 0.001): "21b85d9c20e8c848",
}


@pytest.mark.parametrize("dim,block", [(2, 16), (2, 8), (2, 12), (3, 16), (3, 12)])
@pytest.mark.parametrize("amr", [False, True])
@pytest.mark.parametrize("mu", [0.0, 1e-3])
def test_step_with_gravity_rounds_as_recorded(dim, block, amr, mu):
    assert digest(dim, block, amr, mu, **GRAVITY) == DIGESTS_GRAVITY[dim, block, amr, mu]
