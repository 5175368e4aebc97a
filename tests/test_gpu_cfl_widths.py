"""The CFL bound over the range of cell widths: its FP32 screen divides by the
width with an approximate quotient that is 0 above 2^126.  Widths on both sides
of that, and of 1e30 and 1e-30, the fastest cell among the widest; dt against
the oracle, bit for bit."""
import numpy as np
import pytest

import oracle
import richgpu
import synthetic
from meshview import PackedMesh3D

pytestmark = pytest.mark.gpu

GAMMA = 5 / 3
SCALES = [2.0 ** 126, 1e30, 1.0, 1e-30]


@pytest.mark.parametrize("order", [1, 2])
@pytest.mark.parametrize("moving", [False, True])
@pytest.mark.parametrize("scale", SCALES)
def test_2d(scale, moving, order):
    nx = 24
    side = scale * nx * np.sqrt(np.pi)
    mesh = synthetic.lattice_mesh(nx, nx, (0.0, side, 0.0, side), "rigid", seed=3, jitter=0.05)
    width = np.sqrt(mesh.volume / np.pi)
    assert (width > 1.001 * scale).any() and (width < 0.999 * scale).any()
    rng = np.random.default_rng(4)
    n = mesh.n_cells
    cells = np.stack([np.ones(n), np.full(n, 0.6), *rng.normal(0, 0.1, (2, n))], 1)
    cells[np.argsort(width)[-20:], 2] = np.linspace(40.0, 50.0, 20)
    ev = rng.normal(0, 0.05, (mesh.n_faces, 2)) * moving
    with richgpu.Handle(gamma=GAMMA, order=order, ghost_kind=0, device=0) as h:
        h.upload_mesh(mesh)
        h.set_edge_velocities(ev)
        h.set_cells(cells)
        assert h.cfl_dt() == oracle.cfl(mesh, cells, ev, GAMMA)


@pytest.mark.parametrize("scale", SCALES)
def test_3d(scale):
    nx, ny, nz = 9, 8, 7
    m = synthetic.cube_grid(nx, ny, nz)
    a = {k: np.array(getattr(m, k)) for k in ("face_cells", "face_normal", "face_area", "volume", "width",
                                              "cell_face_offset", "cell_faces")}
    rng = np.random.default_rng(5)
    n = len(a["width"])
    a["width"] = scale * rng.uniform(0.95, 1.05, n)
    mesh = PackedMesh3D(**a)
    cells = np.stack([np.ones(n), np.full(n, 0.6), *rng.normal(0, 0.1, (3, n))], 1)
    cells[np.argsort(a["width"])[-20:], 2] = np.linspace(40.0, 50.0, 20)
    want = oracle.cfl3(mesh, cells, GAMMA)
    with richgpu.Handle3(gamma=GAMMA, device=0) as h:
        h.upload_mesh(mesh)
        h.set_cells(cells)
        assert h.cfl_dt() == want
