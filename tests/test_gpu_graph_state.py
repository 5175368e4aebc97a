"""rg_run_graph against rg_run where the handle's state changes between two
graph runs in a way the captured step depends on: face velocities that leave
(or come to) rest, and device buffers handed out to a caller who then writes
the state.  Bit for bit, for every form of the step (both precisions, both
orders, Heun, batches).
"""
import numpy as np
import pytest

import oracle
import richgpu
import synthetic
from test_gpu_batch import init_ext
from test_oracle_golden import exact

pytestmark = pytest.mark.gpu

GAMMA = 5 / 3


def problem(batch):
    """(mesh, offsets, gammas, cells, extensives) of a lattice or a batch."""
    if batch:
        mesh, off, gam, cells, _ = synthetic.riemann_batch(7, seed=3, min_cells=64, max_cells=900)
        return mesh, off, gam, cells, init_ext(mesh, cells, off, gam)
    mesh = synthetic.lattice_mesh(31, 23, (0.0, 1.0, 0.0, 1.0), "rigid", seed=5)
    rng = np.random.default_rng(6)
    n = mesh.n_cells
    cells = np.stack([np.exp(rng.normal(0, 0.1, n)), np.exp(rng.normal(0, 0.1, n)), *rng.normal(0, 0.2, (2, n))], 1)
    return mesh, None, None, cells, oracle.init_extensives(mesh, cells, GAMMA)


# (precision, order, heun, batch); a first-order batch and an FP64 one too
FORMS = [(p, o, t, b) for p in (0, 1) for o in (1, 2) for t in (0, 1) for b in (False, True)]


def outcome(form, script):
    """The state after `script(handle, advance, mesh, cells, ext)`, once with
    advance = run_graph and once with run."""
    precision, order, heun, batch = form
    mesh, off, gam, cells, ext = problem(batch)
    outs = []
    for graph in (True, False):
        with richgpu.Handle(gamma=GAMMA, order=order, ghost_kind=0, precision=precision, device=0,
                            time_integrator=heun) as h:
            h.upload_mesh(mesh)
            if batch:
                h.set_problems(off, gam)
            h.set_edge_velocities(np.zeros((mesh.n_faces, 2)))
            h.set_cells(cells)
            h.set_extensives(ext)
            script(h, h.run_graph if graph else h.run, mesh, cells, ext)
            outs.append((h.get_cells(), h.get_extensives()) + (tuple(h.problem_times()) if batch else ()))
    return outs


def same(form, script):
    got, want = outcome(form, script)
    for a, b in zip(got, want):
        exact(a, b)


@pytest.mark.parametrize("form", FORMS)
def test_face_velocities_set_between_graph_runs(form):
    def script(h, advance, mesh, cells, ext):
        ev = np.random.default_rng(7).normal(0, 0.3, (mesh.n_faces, 2))
        for w in (ev, np.zeros_like(ev), ev):
            advance(3)
            h.set_edge_velocities(w)
        advance(4)

    same(form, script)


@pytest.mark.parametrize("form", FORMS)
def test_device_buffers_taken_between_graph_runs(form):
    def script(h, advance, mesh, cells, ext):
        advance(3)
        h.device_buffers()
        hot = cells * np.array([1.0, 9.0, 1.0, 1.0])
        heat = np.array([1.0, 3.0, 1.0, 1.0])
        h.set_cells(hot)
        h.set_extensives(ext * heat)
        advance(3)

    same(form, script)


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("order", [1, 2])
def test_point_motion_between_graph_runs(order, precision):
    def script(h, advance, mesh, cells, ext):
        h.set_point_motion(kind=1)
        advance(3)
        h.point_velocities()
        advance(4)

    same((precision, order, 0, False), script)
