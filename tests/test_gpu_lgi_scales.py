"""The FP64 slopes where one cell's neighbours differ by 40 orders of magnitude
and more: the shocked limiter's factor is then far below the normal floats, and
the FP32 screen has to leave its candidates to FP64.  Tracer slopes and fluxes
against the oracle, bit for bit."""
import numpy as np
import pytest

import oracle
import richgpu
from test_gpu_lgi_lanes import GAMMA, MESHES

pytestmark = pytest.mark.gpu


def state(mesh, low, high, seed):
    """Cells shocked by their pressures; tracers of zeros, values around `low`
    and values around `high`, and y velocities of the same kind."""
    rng = np.random.default_rng(seed)
    n = mesh.n_cells
    mixed = rng.choice([0.0, low, high], (n, 4)) * rng.uniform(-2, 2, (n, 4))
    c = np.ones((n, 4))
    c[:, 1] = 10.0 ** rng.uniform(-2, 2, n)
    c[:, 2] = 0.0
    c[:, 3] = mixed[:, 3] / high * 10.0
    return c, mixed[:, :3]


@pytest.mark.parametrize("which", sorted(MESHES))
@pytest.mark.parametrize("low,high", [(1e-29, 1e19), (1e-25, 1e8), (1e-29, 1e36), (1e-10, 1e25), (1e-35, 1.0)])
def test_shocked_limiter_over_mixed_scales(which, low, high):
    mesh, ghost = MESHES[which]()
    cells, tr = state(mesh, low, high, 11)
    stickers = np.zeros(mesh.n_cells, dtype=np.uint32)
    ev = np.zeros((mesh.n_faces, 2))
    lp = oracle.lgi_params(ghost)
    ts = oracle.TracerSetup(3, limited=7, stickers=stickers)
    want_slopes = oracle.lgi_tr(mesh, cells, tr, GAMMA, lp, ts)[2].reshape(-1)
    with richgpu.Handle(gamma=GAMMA, order=2, ghost_kind=ghost) as h:
        h.upload_mesh(mesh)
        h.set_tracer_config(3, limited=[0, 1, 2])
        h.set_cells(cells)
        h.set_tracers(tr)
        h.set_edge_velocities(ev)
        got = h.flux(0.0)
        slopes = h.tracer_slopes().reshape(-1)
    assert np.array_equal(slopes, want_slopes)
    assert np.array_equal(got, oracle.flux_tr(mesh, cells, tr, ev, GAMMA, 2, lp, ts)[0])
