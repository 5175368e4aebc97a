"""The dt a step's update forms for the next one, against the CFL pass: a run of
k steps gives the dts and states of k one-step runs of fresh handles, each of
which starts with the pass, bit for bit (both precisions, first and second
order, 2D and 3D, fewer and more cells than a block's threads)."""
import numpy as np
import pytest

import oracle
import richgpu
import synthetic
from meshview import PackedMesh3D
from test_oracle_golden import exact

pytestmark = pytest.mark.gpu

GAMMA = 5 / 3


def one_by_one(fresh, cells, ext, steps):
    dts = []
    for _ in range(steps):
        with fresh() as h:
            h.set_cells(cells)
            h.set_extensives(ext)
            dts.append(h.run(1)[0])
            cells, ext = h.get_cells(), h.get_extensives()
    return np.array(dts), cells, ext


def check(fresh, cells, ext, steps=6):
    want = one_by_one(fresh, cells, ext, steps)
    with fresh() as h:
        # another state first: its next dt must not reach the run
        h.set_cells(cells * 1.5)
        h.set_extensives(ext * 1.5)
        h.run(2)
        h.set_cells(cells)
        h.set_extensives(ext)
        got = np.asarray(h.run(steps)), h.get_cells(), h.get_extensives()
    for a, b in zip(got, want):
        exact(a, b)


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("order", [1, 2])
@pytest.mark.parametrize("nx,ny,moving", [(5, 7, False), (17, 16, True), (61, 43, True)])
def test_2d(nx, ny, moving, order, precision):
    mesh = synthetic.lattice_mesh(nx, ny, (0.0, 1.0, 0.0, 1.0), "rigid", seed=nx)
    rng = np.random.default_rng(ny)
    n = mesh.n_cells
    cells = np.stack([np.exp(rng.normal(0, 0.1, n)), np.exp(rng.normal(0, 0.1, n)), *rng.normal(0, 0.2, (2, n))], 1)
    if precision:
        cells = cells.astype(np.float32).astype(np.float64)
    ext = oracle.init_extensives(mesh, cells, GAMMA)
    ev = rng.normal(0, 0.05, (mesh.n_faces, 2)) * moving

    def fresh():
        h = richgpu.Handle(gamma=GAMMA, order=order, ghost_kind=0, precision=precision, device=0)
        h.upload_mesh(mesh)
        h.set_edge_velocities(ev)
        return h

    check(fresh, cells, ext)


def grid3(nx, ny, nz, kind):
    """The CubeGrid; "flipped": a third of the faces turned round; "turned": the
    whole grid turned, so that no normal lies on an axis."""
    m = synthetic.cube_grid(nx, ny, nz)
    a = {k: np.array(getattr(m, k)) for k in ("face_cells", "face_normal", "face_area", "volume", "width",
                                              "cell_face_offset", "cell_faces")}
    if kind == "flipped":
        a["face_normal"][::3] *= -1.0
        a["face_cells"][::3] = a["face_cells"][::3, ::-1]
    if kind == "turned":
        q, _ = np.linalg.qr(np.random.default_rng(2).normal(size=(3, 3)))
        a["face_normal"] = a["face_normal"] @ q
    return PackedMesh3D(**a)


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("kind", ["grid", "flipped", "turned"])
@pytest.mark.parametrize("nx,ny,nz", [(3, 4, 5), (9, 8, 7)])
def test_3d(nx, ny, nz, kind, precision):
    mesh = grid3(nx, ny, nz, kind)
    cells = synthetic.cube_blast_cells(nx, ny, nz)
    if precision:
        cells = cells.astype(np.float32).astype(np.float64)
    ext = oracle.init_extensives3(mesh, cells, GAMMA)

    def fresh():
        h = richgpu.Handle3(gamma=GAMMA, device=0, precision=precision)
        h.upload_mesh(mesh)
        return h

    check(fresh, cells, ext)


@pytest.mark.parametrize("kind", ["grid", "flipped", "turned"])
@pytest.mark.parametrize("rest", [False, True])
def test_3d_faces_vs_oracle(kind, rest):
    """Face normals on an axis, either way round, and off it; fluid at rest."""
    nx, ny, nz = 7, 6, 5
    mesh = grid3(nx, ny, nz, kind)
    cells = synthetic.cube_blast_cells(nx, ny, nz)
    if rest:
        cells[:, 2:5] = 0.0
    ext = oracle.init_extensives3(mesh, cells, GAMMA)
    with richgpu.Handle3(gamma=GAMMA, device=0) as h:
        h.upload_mesh(mesh)
        h.set_cells(cells)
        h.set_extensives(ext)
        dts = h.run(6)
        gc, ge = h.get_cells(), h.get_extensives()
    oc, oe, odts = oracle.run3(mesh, cells, ext, GAMMA, 6)
    exact(dts, odts)
    exact(ge, oe)
    exact(gc, oc)
