"""The time steps of the solver loop against the CFL reduction of the states it passes through: a maximum cleared late, lost
or taken from another step shows as a wrong dt, also where the loop and its replay by single steps would agree."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from godunov_mhd_ct_gb300 import workloads as wl  # noqa: E402
from godunov_mhd_ct_gb300.mesh import BlockMesh  # noqa: E402
from godunov_mhd_ct_gb300.solver import GodunovImplemGB300  # noqa: E402

from .helpers import settings  # noqa: E402

pytestmark = pytest.mark.gpu

# FP32 CFL of the mixed loop: some 32 roundings of 2^-24 on an energy up to 30 times the thermal one, halved by the square root
RTOL = {"fp64": 0.0, "mixed": 3e-5}


def _uniform(dim, level, block, **kw):
    mesh = BlockMesh.uniform(dim, level=level, block=(block, block, block if dim == 3 else 1), **kw)
    return mesh, wl.random_smooth(mesh, seed=5), {}


def _batch():
    meshes, states, _ = wl.field_loop_batch(5, seed=2, sizes=(32, 64))
    mesh, problem = BlockMesh.batch(meshes)
    return mesh, (np.concatenate([s[0] for s in states]), np.concatenate([s[1] for s in states])), \
        {"problem": problem, "n_problems": len(meshes)}


def _amr():
    mesh = BlockMesh.amr(2, wl.refine_band((0.5, 0.5, 0.5), 0.15, 0.25), base_level=2, max_level=4, block=(16, 16, 1))
    return mesh, wl.random_smooth(mesh, seed=5), {}


CASES = {
    "2d_one_tile": lambda: _uniform(2, 0, 16),
    "2d_64_tiles": lambda: _uniform(2, 3, 16),
    "2d_waves": lambda: _uniform(2, 5, 16),
    "2d_walls": lambda: (*_uniform(2, 2, 16, periodic=(True, False, True))[:2], {"bc": (1, 1, 3, 3, 1, 1)}),
    "3d": lambda: _uniform(3, 2, 16),
    "3d_b12": lambda: _uniform(3, 1, 12),
    "batch": _batch,
    "2d_amr": _amr,
}


@pytest.mark.parametrize("name", sorted(CASES))
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("ends", [False, True])
def test_time_steps_follow_the_states(name, precision, ends):
    mesh, (U, B), kw = CASES[name]()
    st = settings(cfl=0.4)
    impl = GodunovImplemGB300(st, mesh, precision=precision, **kw)
    npb, nsteps = kw.get("n_problems", 1), 5

    def loop(k, t_end, graph=True):
        u, b = torch.from_numpy(U).cuda(), torch.from_numpy(B).cuda()
        dts, t = impl.advance(u, torch.zeros_like(u), b, torch.zeros_like(b), k, t=0.0, t_end=t_end, use_graph=graph)
        return dts, t, u, b

    t_end = None
    if ends:  # some problems end inside the loop, the others after it
        t_end = loop(nsteps, None)[1] * np.linspace(0.5, 1.5, npb) if npb > 1 else loop(nsteps, None)[1] * 0.7
    dts, t, _, _ = loop(nsteps, t_end)
    assert np.array_equal(loop(nsteps, t_end, graph=False)[0], dts)
    at = np.zeros(npb)
    for k in range(nsteps):
        _, tk, u, b = loop(k, t_end) if k else (None, at.copy(), torch.from_numpy(U).cuda(), torch.from_numpy(B).cuda())
        assert np.array_equal(tk, at)
        want = st.cfl / np.atleast_1d(impl.compute_inv_dt(u, b))
        if ends:
            left = np.broadcast_to(t_end, (npb,)) - at
            want = np.where(left > 0.0, np.minimum(want, left), 0.0)
        assert np.all(np.abs(dts[k] - want) <= RTOL[precision] * want), (k, dts[k], want)
        at = at + dts[k]
    assert np.array_equal(t, at)
    impl.close()
