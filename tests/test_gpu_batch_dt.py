"""The dt that a batch's step returns is problem 0's, as rg_run's record has it:
rg_step, rg_step_timed, rg_step_async + rg_synchronize, and rg_synchronize after
a persistent run, for both precisions and orders and Heun."""
import numpy as np
import pytest

import richgpu
import synthetic
from test_gpu_batch import init_ext
from test_oracle_golden import exact

pytestmark = pytest.mark.gpu


def handle(batch, precision, order, heun):
    mesh, off, gam, cells, ext = batch
    h = richgpu.Handle(gamma=1.4, order=order, ghost_kind=0, precision=precision, device=0, time_integrator=heun)
    h.upload_mesh(mesh)
    h.set_problems(off, gam)
    h.set_edge_velocities(np.zeros((mesh.n_faces, 2)))
    h.set_cells(cells)
    h.set_extensives(ext)
    return h


@pytest.fixture(scope="module")
def batch():
    mesh, off, gam, cells, _ = synthetic.riemann_batch(5, seed=3, min_cells=64, max_cells=900)
    return mesh, off, gam, cells, init_ext(mesh, cells, off, gam)


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("order,heun", [(1, 0), (2, 0), (2, 1)])
def test_step_returns_problem_0s_dt(batch, precision, order, heun):
    with handle(batch, precision, order, heun) as h:
        want = h.run(4)
    with handle(batch, precision, order, heun) as h:
        got = [h.step(), h.step_timed()[0]]
        assert h.problem_times()[1][0] == got[1]
        h.step_async()
        got.append(h.synchronize())
        h.run(1)
        got.append(h.synchronize())
    exact(np.array(got), want)


def test_after_a_persistent_run(batch):
    with handle(batch, 1, 2, 0) as h:
        h.set_step_mode(richgpu.STEP_PERSISTENT)
        dts = h.run(3)
        assert h.synchronize() == dts[-1]
