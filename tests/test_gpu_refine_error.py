"""The block error of the refinement indicator is the exact maximum of its quotients: against the same formulas in numpy,
bit for bit, by thresholds at the error itself and one unit below it. Blocks smaller than, equal to and not a multiple of a
CTA's 256 cells; values of ordinary size, over 600 orders of magnitude, and with zeros, infinities and NaN."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from godunov_mhd_ct_gb300.mesh import BlockMesh  # noqa: E402
from godunov_mhd_ct_gb300.solver import GodunovImplemGB300  # noqa: E402

from .helpers import settings  # noqa: E402

pytestmark = pytest.mark.gpu

EPS = 0.02


def _errors(rho, dim, criterion):
    v = rho
    quotients = []
    with np.errstate(all="ignore"):
        for d in range(dim):
            ax = 3 - d
            edge = [slice(None)] * 4
            edge[ax] = slice(0, 1)
            qm = np.concatenate([v[tuple(edge)], np.delete(v, -1, ax)], ax)
            edge[ax] = slice(-1, None)
            qp = np.concatenate([np.delete(v, 0, ax), v[tuple(edge)]], ax)
            if criterion == "SIMPLE_GRADIENT":
                e = np.fmax(np.abs(qp - v), np.abs(v - qm)) / np.fmax(np.abs(v), np.finfo(np.float64).tiny)
            else:
                dp, dm = qp - v, v - qm
                den = np.abs(dp) + np.abs(dm) + EPS * (np.abs(qp) + 2.0 * np.abs(v) + np.abs(qm))
                e = np.where(den > 0.0, np.abs(dp - dm) / den, 0.0)
            quotients.append(e)
    return np.fmax.reduce(np.stack(quotients).transpose(1, 0, 2, 3, 4).reshape(v.shape[0], -1), axis=1, initial=0.0)


@pytest.mark.parametrize("dim,block", [(2, 4), (2, 16), (2, 20), (3, 4), (3, 8), (3, 12)])
@pytest.mark.parametrize("criterion", ["SIMPLE_GRADIENT", "LOHNER_UNSPLIT"])
@pytest.mark.parametrize("kind", ["plain", "wide", "special"])
def test_block_error_is_exact(dim, block, criterion, kind):
    mesh = BlockMesh.uniform(dim, level=1, block=(block, block, block if dim == 3 else 1))
    U, B = mesh.alloc_state()
    rng = np.random.default_rng(block + dim)
    rho = rng.uniform(0.5, 1.5, U[:, 0].shape)
    if kind == "wide":
        rho = rho * 10.0 ** rng.integers(-300, 300, rho.shape)
    if kind == "special":
        pick = rng.integers(0, 60, rho.shape)
        for n, x in enumerate((0.0, -0.0, np.inf, np.nan, 1e-310, -2.0)):
            rho[pick == n] = x
    U[:, 0] = rho
    err = _errors(rho[: mesh.n_owned], dim, criterion)
    impl = GodunovImplemGB300(settings(), mesh, precision="fp64")
    dU, dB = torch.from_numpy(U).cuda(), torch.from_numpy(B).cuda()
    for n, e in enumerate(err):
        for eps, flag in ((e, 0), (np.nextafter(e, 0.0), 1 if e > 0.0 else 0)):
            f = impl.refine_flags(dU, dB, criterion=criterion, level_min=0, level_max=2, eps_refine=float(eps),
                                  eps_coarsen=0.0, eps_lohner=EPS, variables=("rho",))
            assert f[n] == flag, (n, e, eps)
    impl.close()
