"""Cells without faces, the smallest mesh an upload accepts: the dts a run
records are those of the same steps on fresh handles (whose every step forms its
dt in a CFL pass), at both orders and precisions."""
import numpy as np
import pytest

import oracle
import richgpu
from meshview import PackedMesh
from test_oracle_golden import exact

pytestmark = pytest.mark.gpu

GAMMA = 5 / 3


def mesh_of(n):
    x = np.arange(2.0 * n).reshape(n, 2)
    return PackedMesh(point_xy=x, cm_xy=x, volume=np.ones(n), cd_volume=np.ones(n), ghost_source=np.zeros(0, np.int32),
                      ghost_face=np.zeros(0, np.int32), face_cells=np.zeros((0, 2), np.int32),
                      face_vertices=np.zeros((0, 4)), cell_face_offset=np.zeros(n + 1, np.int32),
                      cell_faces=np.zeros(0, np.int32))


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("order", [1, 2])
@pytest.mark.parametrize("n", [1, 3])
def test_run_records_every_dt(n, order, precision):
    mesh = mesh_of(n)
    cells = np.stack([np.full(n, 1.0), 1.0 + np.arange(n), np.zeros(n), np.zeros(n)], 1)
    ext = oracle.init_extensives(mesh, cells, GAMMA)

    def fresh(c, u):
        h = richgpu.Handle(gamma=GAMMA, order=order, ghost_kind=0, precision=precision, device=0)
        h.upload_mesh(mesh)
        h.set_edge_velocities(np.zeros((0, 2)))
        h.set_cells(c)
        h.set_extensives(u)
        return h

    want, c, u = [], cells, ext
    for _ in range(4):
        with fresh(c, u) as h:
            want.append(h.run(1)[0])
            c, u = h.get_cells(), h.get_extensives()
    with fresh(cells, ext) as h:
        got = np.concatenate([h.run(3), [h.step()]])
        exact(h.get_cells(), c)
        exact(h.get_extensives(), u)
    assert np.array_equal(got, want)  # (an infinite dt is the reference's for FP64: no face bounds it)
