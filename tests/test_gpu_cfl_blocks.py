"""The CFL reduction finds the fastest cell wherever it lies: blocks whose length does not divide a CTA's 256 cells, and cells
at the ends of a thread's, a chunk's (1024 cells) and the block's range."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from godunov_mhd_ct_gb300 import workloads as wl  # noqa: E402
from godunov_mhd_ct_gb300.mesh import BlockMesh  # noqa: E402
from godunov_mhd_ct_gb300.solver import GodunovImplemGB300  # noqa: E402

from .helpers import oracle_mesh, oracle_settings, settings  # noqa: E402
from .test_zz_no_alloc import _noalloc  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,block,level", [(2, (12, 12, 1), 2), (2, (20, 20, 1), 1), (2, (36, 36, 1), 1), (2, (12, 20, 1), 1),
                                             (2, (260, 260, 1), 0), (3, (12, 12, 12), 1), (3, (20, 20, 20), 0),
                                             (3, (36, 36, 36), 0), (3, (12, 20, 36), 0), (3, (4, 4, 4), 1)])
def test_fastest_cell_anywhere(oracle_lib, dim, block, level):
    mesh = BlockMesh.uniform(dim, level=level, block=block)
    st = settings(cfl=0.4)
    U, B = wl.random_smooth(mesh, gamma=st.gamma0, seed=block[0])
    om, os_ = oracle_mesh(oracle_lib, mesh), oracle_settings(oracle_lib, st)
    exact = GodunovImplemGB300(st, mesh, precision="fp64")
    mixed = GodunovImplemGB300(st, mesh, precision="mixed")
    ncell = int(np.prod(block))
    rng = np.random.default_rng(1)
    cells = {0, 255, 256, 257, 511, 512, 1023, 1024, ncell - 1, block[0] - 1, *rng.integers(0, ncell, 6).tolist()}
    slowest = exact.compute_inv_dt(torch.from_numpy(U).cuda(), torch.from_numpy(B).cuda())
    for n, c in enumerate(sorted(x for x in cells if x < ncell)):
        V = U.copy()
        cell = V[n % mesh.n_owned].reshape(5, -1)[:, c]  # a view
        k = rng.integers(2, 2 + dim)
        cell[1] -= 0.5 * cell[k] ** 2 / cell[0]
        cell[k] = 8.0 * cell[0]
        cell[1] += 0.5 * cell[k] ** 2 / cell[0]
        dV, dB = torch.from_numpy(V).cuda(), torch.from_numpy(B).cuda()
        want = oracle_lib.inv_dt(om, os_, V, B)
        assert want > 1.2 * slowest
        assert exact.compute_inv_dt(dV, dB) == want, c
        assert _noalloc(st, mesh, dV, dB)[0] == want, c
        # the mixed loop's first step: FP32, some 32 roundings of 2^-24 on an energy 60 times the thermal one
        dts, _ = mixed.advance(dV, torch.zeros_like(dV), dB, torch.zeros_like(dB), 1)
        assert abs(dts[0, 0] * want / st.cfl - 1.0) <= 6e-5, c
    exact.close()
    mixed.close()
