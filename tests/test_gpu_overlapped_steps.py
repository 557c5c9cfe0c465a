"""The solver loop starts each kernel while the one before drains. Its states must be those of the same time steps taken
one call at a time, bit for bit: meshes of one tile, of fewer tiles than SMs and of several waves, every kernel family,
coarse/fine passes, and outside blocks filled between the kernels."""
import pytest

torch = pytest.importorskip("torch")

from godunov_mhd_ct_gb300 import workloads as wl  # noqa: E402
from godunov_mhd_ct_gb300.mesh import BlockMesh  # noqa: E402
from godunov_mhd_ct_gb300.solver import GodunovImplemGB300  # noqa: E402

from .helpers import settings  # noqa: E402

pytestmark = pytest.mark.gpu

MESHES = {
    "2d_one_tile": lambda: BlockMesh.uniform(2, level=0, block=(16, 16, 1)),
    "2d_64_tiles": lambda: BlockMesh.uniform(2, level=3, block=(16, 16, 1)),
    "2d_walls": lambda: BlockMesh.uniform(2, level=2, block=(16, 16, 1), periodic=(True, False, True)),
    "2d_waves": lambda: BlockMesh.uniform(2, level=5, block=(16, 16, 1)),
    "3d": lambda: BlockMesh.uniform(3, level=2, block=(16, 16, 16)),
    "3d_b4": lambda: BlockMesh.uniform(3, level=2, block=(4, 4, 4)),
    "2d_amr": lambda: BlockMesh.amr(2, wl.refine_band((0.5, 0.5, 0.5), 0.15, 0.25), base_level=2, max_level=4, block=(16, 16, 1)),
    "3d_amr": lambda: BlockMesh.amr(3, wl.refine_band((0.3, 0.3, 0.3), 0.0, 0.2, axes=3), base_level=1, max_level=2,
                                    block=(8, 8, 8)),
}


@pytest.mark.parametrize("name,precision,tile", [(n, p, 0) for n in MESHES for p in ("mixed", "fp64")]
                         + [("3d", "mixed", 16)])
def test_advance_equals_single_steps(name, precision, tile):
    mesh = MESHES[name]()
    st = settings(gamma0=1.4, cfl=0.4)
    U, B = wl.random_smooth(mesh, seed=3)
    bc = (1, 1, 3, 3, 1, 1) if name == "2d_walls" else None
    impl = GodunovImplemGB300(st, mesh, precision=precision, **({"bc": bc} if bc else {}))
    if tile:
        impl.set_tile(tile)
    for nsteps, graph in ((6, True), (5, True), (5, False)):
        u, b = torch.from_numpy(U).cuda(), torch.from_numpy(B).cuda()
        dts, _ = impl.advance(u, torch.zeros_like(u), b, torch.zeros_like(b), nsteps, use_graph=graph)
        v, c = torch.from_numpy(U).cuda(), torch.from_numpy(B).cuda()
        v2, c2 = torch.zeros_like(v), torch.zeros_like(c)
        for dt in dts[:, 0]:
            impl.fill_outside(v, c)
            impl.do_time_step(v, v2, c, c2, float(dt))
            v, v2, c, c2 = v2, v, c2, c
        n = mesh.n_owned
        assert torch.equal(u[:n], v[:n]) and torch.equal(b[:n], c[:n]), (nsteps, graph)
    impl.close()
