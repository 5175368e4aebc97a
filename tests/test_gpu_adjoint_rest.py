"""rg_step_fwd on a handle that was given no face velocities: the faces are at
rest, whatever the memory held before (it read the unset buffer)."""
import numpy as np
import pytest

import richgpu
import synthetic
from test_oracle_golden import exact

pytestmark = pytest.mark.gpu

GAMMA = 5 / 3


def handle(mesh, precision):
    h = richgpu.Handle(gamma=GAMMA, order=2, ghost_kind=1, precision=precision, device=0)
    h.upload_mesh(mesh)
    return h


@pytest.mark.parametrize("precision", [0, 1])
def test_unset_face_velocities_are_zero(precision):
    mesh = synthetic.lattice_mesh(33, 21, (0.0, 1.0, 0.0, 1.0), "periodic", seed=5)
    cells = synthetic.bumps_cells(mesh)
    wbar = np.random.default_rng(1).normal(size=cells.shape)
    out = []
    for given in (True, False, False, False):
        # memory of the same sizes that held large velocities, given back
        dirty = [handle(mesh, precision) for _ in range(3)]
        for h in dirty:
            h.set_edge_velocities(np.full((mesh.n_faces, 2), 1e6))
            h.close()
        with handle(mesh, precision) as h:
            if given:
                h.set_edge_velocities(np.zeros((mesh.n_faces, 2)))
            h.set_cells(cells)
            h.step_fwd(4, 1e-4, 2)
            out.append((h.get_cells(), h.step_bwd(wbar)))
    for c, g in out[1:]:
        exact(c, out[0][0])
        exact(g, out[0][1])
