"""Steps after a rejected cell (negative thermal energy).  The cell keeps its
record, so the dt a fused step's update forms for the next one has to count it
as the CFL pass over the records does: fused runs against steps that each begin
with the pass, bit for bit, the rejected cell being the one that sets the dt.
"""
import numpy as np
import pytest

import oracle
import richgpu
import synthetic
from richgpu import dptr
from test_gpu_batch import init_ext
from test_oracle_golden import exact

pytestmark = pytest.mark.gpu

GAMMA = 5 / 3
NEGATIVE_ENERGY = 11


def run(h, steps):
    """The dts of `steps` steps, of which at least one rejects a cell."""
    dts = np.full(steps, -1.0)
    fn = h.lib.rg3_run if isinstance(h, richgpu.Handle3) else h.lib.rg_run
    assert fn(h.h, steps, dptr(dts)) == NEGATIVE_ENERGY
    return dts


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("order", [1, 2])
def test_2d(order, precision):
    mesh = synthetic.lattice_mesh(23, 19, (0.0, 1.0, 0.0, 1.0), "rigid", seed=2)
    rng = np.random.default_rng(3)
    n = mesh.n_cells
    cells = np.stack([np.exp(rng.normal(0, 0.1, n)), np.exp(rng.normal(0, 0.1, n)), *rng.normal(0, 0.1, (2, n))], 1)
    bad = 217
    ext = oracle.init_extensives(mesh, cells, GAMMA)
    cells[bad, 1] = 40.0  # the largest sound speed
    ext[bad, 1] = -50.0
    outs = []
    for fused in (True, False):
        with richgpu.Handle(gamma=GAMMA, order=order, ghost_kind=0, precision=precision, device=0) as h:
            h.upload_mesh(mesh)
            if not fused:
                h.device_buffers()  # steps with a CFL pass of their own
            h.set_edge_velocities(np.zeros((mesh.n_faces, 2)))
            h.set_cells(cells)
            h.set_extensives(ext)
            dts = [run(h, 3), run(h, 1), run(h, 2)]
            outs.append((np.concatenate(dts), h.get_cells(), h.get_extensives()))
    for a, b in zip(*outs):
        exact(a, b)


@pytest.mark.parametrize("where", [0, 4])
def test_batch(where):
    mesh, off, gam, cells, _ = synthetic.riemann_batch(6, seed=3, min_cells=64, max_cells=900)
    ext = init_ext(mesh, cells, off, gam)
    bad = (off[where] + off[where + 1]) // 2
    cells[bad, 1] *= 50.0
    ext[bad, 1] = -50.0
    outs = []
    for mode in ("fused", "pass", "persistent"):
        with richgpu.Handle(gamma=1.4, order=2, ghost_kind=0, precision=1, device=0) as h:
            h.upload_mesh(mesh)
            h.set_problems(off, gam)
            if mode == "pass":
                h.device_buffers()
            if mode == "persistent":
                h.set_step_mode(richgpu.STEP_PERSISTENT)
            h.set_edge_velocities(np.zeros((mesh.n_faces, 2)))
            h.set_cells(cells)
            h.set_extensives(ext)
            dts = [run(h, 3), run(h, 2)]
            outs.append((np.concatenate(dts), h.get_cells(), h.get_extensives()) + tuple(h.problem_times()))
    for o in outs[1:]:
        for a, b in zip(o, outs[0]):
            exact(a, b)


@pytest.mark.parametrize("precision", [0, 1])
def test_3d(precision):
    nx, ny, nz = 9, 8, 7
    mesh = synthetic.cube_grid(nx, ny, nz)
    cells = synthetic.cube_blast_cells(nx, ny, nz)
    ext = oracle.init_extensives3(mesh, cells, GAMMA)
    bad = 251
    cells[bad, 1] = 50.0 * cells[:, 1].max()
    if precision:
        cells = cells.astype(np.float32).astype(np.float64)
    ext[bad, 0] *= 100.0  # (it stays positive through what the steps take from it)
    ext[bad, 4] = -50.0

    def fresh(c, u):
        h = richgpu.Handle3(gamma=GAMMA, device=0, precision=precision)
        h.upload_mesh(mesh)
        h.set_cells(c)
        h.set_extensives(u)
        return h

    want, c, u = [], cells, ext
    for _ in range(5):
        with fresh(c, u) as h:
            want.append(run(h, 1)[0])
            c, u = h.get_cells(), h.get_extensives()
    with fresh(cells, ext) as h:
        got = np.concatenate([run(h, 3), run(h, 2)])
        exact(h.get_cells(), c)
        exact(h.get_extensives(), u)
    exact(got, np.array(want))
