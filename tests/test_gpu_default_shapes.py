"""The launch shapes of a new handle as a base for others: any block size set
beside the reported build is accepted, for every kernel, and gives the same
results."""
import ctypes as C

import numpy as np
import pytest

import richgpu
from test_gpu_tune import sedov
from test_oracle_golden import exact

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("block", [64, 256, 512])
def test_reported_builds_take_every_block(block, precision):
    mesh, cells, ext = sedov(48)
    outs = []
    for changed in (False, True):
        with richgpu.Handle(gamma=5 / 3, order=2, ghost_kind=0, precision=precision, device=0) as h:
            h.upload_mesh(mesh)
            if changed:
                r = richgpu.RgLaunchShapes()
                assert h.lib.rg_get_launch_shapes(h.h, C.byref(r)) == 0
                for k in range(4):
                    r.block[k] = block
                assert h.lib.rg_set_launch_shapes(h.h, C.byref(r)) == 0
            h.set_cells(cells)
            h.set_extensives(ext)
            h.set_edge_velocities(np.zeros((mesh.n_faces, 2)))
            outs.append((h.run(5), h.get_cells(), h.get_extensives()))
    for a, b in zip(*outs):
        exact(a, b)
