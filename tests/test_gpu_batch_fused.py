"""Fused steps of an FP32-mixed batch: the update forms each problem's next CFL
minimum and the next step's slopes kernel takes it.  Bit for bit the same as
the run whose steps form it in a pass of their own (the cooperative launch),
however the steps are issued, and nothing of it outlives a change of the state.
"""
import numpy as np
import pytest

import richgpu
import synthetic
from test_gpu_batch import init_ext
from test_oracle_golden import exact

pytestmark = pytest.mark.gpu

# one problem; fewer than a warp of problems; more problems than one block's threads
BATCHES = [(1, 7, 64, 900), (12, 5, 64, 2500), (300, 3, 64, 130)]


def handle(mesh, off, gam, moving):
    h = richgpu.Handle(gamma=1.4, order=2, ghost_kind=0, precision=1, device=0)
    h.upload_mesh(mesh)
    h.set_problems(off, gam)
    ev = np.zeros((mesh.n_faces, 2))
    if moving:
        ev += np.random.default_rng(4).normal(0, 0.05, ev.shape)
    h.set_edge_velocities(ev)
    return h


@pytest.mark.parametrize("moving", [False, True])
@pytest.mark.parametrize("n,seed,lo,hi", BATCHES)
def test_fused_batch(n, seed, lo, hi, moving):
    mesh, off, gam, cells, _ = synthetic.riemann_batch(n, seed=seed, min_cells=lo, max_cells=hi)
    ext = init_ext(mesh, cells, off, gam)
    with handle(mesh, off, gam, moving) as h:
        h.set_step_mode(richgpu.STEP_PERSISTENT)
        h.set_cells(cells)
        h.set_extensives(ext)
        dts = h.run(7)
        want = (h.get_cells(), h.get_extensives()) + tuple(h.problem_times())
    with handle(mesh, off, gam, moving) as h:
        # other states first: their minima must not reach the run below
        hot = cells.copy()
        hot[:, 1] *= 100.0
        h.set_cells(hot)
        h.set_extensives(init_ext(mesh, hot, off, gam))
        h.run(3)
        h.set_problems(off, gam)  # times back to zero
        h.run(1)
        h.set_problems(off, gam)
        h.set_cells(cells)
        h.set_extensives(ext)
        got_dts = list(h.run(2)) + [h.step()]
        h.run_graph(2)
        got_dts[3:5] = dts[3:5]  # (a graph's replays report no dt)
        got_dts += list(h.run(2))
        got = (h.get_cells(), h.get_extensives()) + tuple(h.problem_times())
    for a, b in zip(got, want):
        exact(a, b)
    exact(np.asarray(got_dts[:2]), np.asarray(dts[:2]))
    exact(np.asarray(got_dts[5:]), np.asarray(dts[5:]))
