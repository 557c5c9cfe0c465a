"""Refinement flags of meshes whose blocks share a CTA (fewer than 256 cells each), fill one or take several: rho and the
pressure against the oracle, with block counts that do not divide into whole CTAs."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from godunov_mhd_ct_gb300 import workloads as wl  # noqa: E402
from godunov_mhd_ct_gb300.mesh import BlockMesh  # noqa: E402
from godunov_mhd_ct_gb300.solver import GodunovImplemGB300  # noqa: E402

from .helpers import oracle_settings, settings  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,bricks,level,block", [(2, 3, 0, 4), (2, 3, 2, 4), (2, 5, 1, 4), (2, 3, 1, 8), (2, 3, 1, 12), (2, 1, 1, 16),
                                                    (2, 3, 0, 20), (3, 3, 0, 4), (3, 3, 1, 4), (3, 1, 1, 8), (3, 1, 0, 12)])
@pytest.mark.parametrize("criterion", ["SIMPLE_GRADIENT", "LOHNER_UNSPLIT"])
def test_flags_of_any_block_size(oracle_lib, dim, bricks, level, block, criterion):
    mesh = BlockMesh.uniform(dim, bricks=(bricks, 1, 1), level=level, block=(block, block, block if dim == 3 else 1))
    st = settings(gamma0=1.4)
    U, B = wl.random_smooth(mesh, seed=block)
    rng = np.random.default_rng(block + level)
    amp = 10.0 ** rng.uniform(-3.0, -0.7, mesh.n_owned)[:, None, None, None]  # some blocks rough, some smooth
    for v in (0, 1):
        U[:, v] *= 1.0 + amp * rng.uniform(-1.0, 1.0, U[:, v].shape)
    impl = GodunovImplemGB300(st, mesh, precision="fp64")
    seen = set()
    for variables in (("rho",), ("pressure",), ("rho", "pressure")):
        for refine, coarsen in ((0.2, 0.05), (0.05, 0.02), (0.6, 0.3)):
            kw = dict(criterion=criterion, level_min=max(level - 1, 0), level_max=level + 1, eps_refine=refine, eps_coarsen=coarsen)
            got = impl.refine_flags(torch.from_numpy(U).cuda(), torch.from_numpy(B).cuda(), variables=variables, **kw)
            want = oracle_lib.refine_flags(oracle_lib.Mesh.from_block_mesh(mesh), oracle_settings(oracle_lib, st), U, B,
                                           use_rho="rho" in variables, use_pressure="pressure" in variables, **kw)
            assert np.array_equal(got, want), (variables, refine)
            seen |= set(want.tolist())
    assert len(seen) > 1 or mesh.n_owned < 8
    impl.close()
