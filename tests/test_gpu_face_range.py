"""The FP64 face kernels' integer forms and their general form (rg_face.cuh,
face_exact) against the oracle, bit for bit: fluid at rest (zero operands in
most products), densities and pressures near both ends of the exponent range
(products and quotients outside the integer forms), scales that change from
cell to cell, moving faces, rigid walls and odd counts.  Equality: every form is
the reference's arithmetic.
"""
import numpy as np
import pytest

import oracle
import richgpu
import synthetic
from test_oracle_golden import exact

pytestmark = pytest.mark.gpu

GAMMA = 5 / 3


def state(mesh, kind, rng):
    n = mesh.n_cells
    c = np.stack([np.exp(rng.normal(0, 0.2, n)), np.exp(rng.normal(0, 0.2, n)), *rng.normal(0, 0.3, (2, n))], 1)
    if kind == "rest":
        c[:, 2:] = 0.0
    elif kind == "uniform":
        c[:] = (1.0, 1.0, 0.5, 0.0)
    elif kind.startswith("2^"):
        c[:, :2] *= 2.0 ** int(kind[2:])
    elif kind == "scales":
        c[:, :2] *= 2.0 ** rng.integers(-40, 40, n)[:, None]
    return c


@pytest.mark.parametrize("order", [1, 2])
@pytest.mark.parametrize("moving", [False, True])
@pytest.mark.parametrize("kind", ["smooth", "rest", "uniform", "2^-1000", "2^-400", "2^300", "2^1000", "scales"])
def test_one_step(kind, moving, order):
    mesh = synthetic.lattice_mesh(13, 11, (0.0, 1.0, 0.0, 1.0), "rigid", seed=3)
    rng = np.random.default_rng(9)
    cells = state(mesh, kind, rng)
    ev = rng.normal(0, 0.1, (mesh.n_faces, 2)) * moving
    ext = oracle.init_extensives(mesh, cells, GAMMA)
    want = err = None
    try:
        want = oracle.run(mesh, cells, ext, ev, GAMMA, 1, 0.3, order, oracle.lgi_params(0))
    except oracle.OracleError as e:  # a state the scheme rejects: then both reject it
        err = e
    with richgpu.Handle(gamma=GAMMA, order=order, ghost_kind=0, device=0) as h:
        h.upload_mesh(mesh)
        h.set_edge_velocities(ev)
        h.set_cells(cells)
        h.set_extensives(ext)
        if err is not None:
            with pytest.raises(richgpu.RichError) as got:
                h.run(1)
            assert got.value.status == err.status
            return
        dts = h.run(1)
        got = h.get_cells(), h.get_extensives(), np.asarray(dts)
    for a, b in zip(got, want):
        exact(a, b)
