"""The FP64 slopes with the limiter's FP32 screen (one lane per component)
against the oracle, bit for bit, where the screen can go wrong: fields flat
to rounding, zero and negative values, ties between faces, extrema, strong
shocks, values near and beyond the range of a float, cells with more
neighbours than the kernel keeps in registers, and odd cell counts (partial
warps and tiles).  The tolerance is equality: the screen only leaves out
candidates that cannot set the limiter's factor.
"""
import numpy as np
import pytest

import oracle
import richgpu
import synthetic
from meshview import PackedMesh

pytestmark = pytest.mark.gpu

GAMMA = 5.0 / 3.0


def random_mesh(n, seed):
    """Periodic Voronoi mesh of n random points in the unit square (cells with
    4 to 12 neighbours), in the packed format."""
    spatial = pytest.importorskip("scipy.spatial")
    rng = np.random.default_rng(seed)
    x = rng.uniform(0, 1, (n, 2))
    shifts = [(0, 0)] + [(i, j) for i in (-1, 0, 1) for j in (-1, 0, 1) if (i, j) != (0, 0)]
    pts = np.concatenate([x + s for s in shifts])
    vor = spatial.Voronoi(pts)
    rows, verts, ghosts = [], [], {}
    for (p, q), rv in zip(vor.ridge_points, vor.ridge_vertices):
        if p >= n and q >= n or min(rv) < 0:
            continue
        v = vor.vertices[rv]
        if np.hypot(*(v[1] - v[0])) < 1e-9:
            continue
        rows.append((p, q))
        verts.append(np.concatenate([v[0], v[1]]))
    order = sorted(range(len(rows)), key=lambda k: (min(rows[k]), max(rows[k])))
    rows, verts = [rows[k] for k in order], np.array([verts[k] for k in order])
    fc, gface = [], []
    for e, (p, q) in enumerate(rows):
        ids = []
        for c in (p, q):
            if c >= n and c not in ghosts:
                ghosts[c] = n + len(ghosts)
                gface.append(e)
            ids.append(c if c < n else ghosts[c])
        fc.append(ids)
    fc = np.array(fc)
    gpts = np.array(sorted(ghosts, key=ghosts.get), dtype=np.int64)
    cells = [[] for _ in range(n)]
    for e, (a, b) in enumerate(fc):
        for c in (a, b):
            if c < n:
                cells[c].append(e)
    off = np.concatenate([[0], np.cumsum([len(c) for c in cells])])
    cf = np.concatenate(cells)
    vol, cm = np.zeros(n), np.zeros((n, 2))
    for i in range(n):
        an, c, a2 = verts[cells[i][0]][:2], np.zeros(2), 0.0
        for e in cells[i]:
            v0, v1 = verts[e][:2], verts[e][2:]
            d0, d1 = v0 - x[i], v1 - x[i]
            vol[i] += 0.5 * abs(d0[0] * d1[1] - d0[1] * d1[0])
            d0, d1 = v0 - an, v1 - an
            t = 0.5 * abs(d0[0] * d1[1] - d0[1] * d1[0])
            a2 += t
            c += (an + v0 + v1) * (t / 3)
        cm[i] = c / a2
    src = gpts % n
    point_xy = np.concatenate([x, pts[gpts]])
    return PackedMesh(point_xy=point_xy, cm_xy=np.concatenate([cm, cm[src] + (pts[gpts] - x[src])]), volume=vol,
                      cd_volume=vol, ghost_source=src, ghost_face=np.array(gface), face_cells=fc, face_vertices=verts,
                      cell_face_offset=off, cell_faces=cf)


MESHES = {
    "rigid": lambda: (synthetic.lattice_mesh(37, 29, (-1, 1, -1, 1), "rigid", seed=1, jitter=0.05), 0),
    "periodic": lambda: (synthetic.lattice_mesh(33, 31, (0, 1, 0, 1), "periodic", seed=2, jitter=1e-3), 1),
    "random": lambda: (random_mesh(397, 3), 1),
}


def field(kind, mesh, rng):
    """(cells, tracer) of one kind of state."""
    n = mesh.n_cells
    x = mesh.point_xy[:n]
    c = np.zeros((n, 4))
    c[:, 0], c[:, 1] = 1.0, 1.0
    noise = rng.uniform(-1, 1, (n, 4))
    t = 1.0 + 0.1 * np.sin(5 * x[:, 0]) * np.cos(4 * x[:, 1])
    if kind == "flat":                      # constant: exact zeros and rounding-level slopes
        t[:] = -0.3
    elif kind == "noise":                   # a plateau with relative noise at and above rounding
        c[:, :2] *= 1.0 + 10.0 ** rng.uniform(-17, -6, (n, 2)) * noise[:, :2]
        c[:, 2:] = 10.0 ** rng.uniform(-30, -9, (n, 2)) * noise[:, 2:]
        t = -1.0 + 10.0 ** rng.uniform(-17, -6, n) * noise[:, 0]
    elif kind == "linear":                  # faces tie
        c[:, 0] += 0.125 * x[:, 0]
        c[:, 1] += 0.25 * x[:, 1]
        c[:, 2] = 0.5 * (x[:, 0] + x[:, 1])
        c[:, 3] = -x[:, 0]
        t = x[:, 0] - x[:, 1]
    elif kind == "steps":                   # exact ties between neighbours, extrema, sign changes
        c += np.round(noise * 2) * [0.25, 0.25, 0.5, 0.5]
        t = np.round(noise[:, 0] * 2)
    elif kind == "shocks":                  # pressure jumps and strong compression
        c[:, 0] *= 10.0 ** noise[:, 0]
        c[:, 1] *= 10.0 ** (2 * noise[:, 1])
        c[:, 2:] = -3.0 * (x - x.mean(0)) + 0.1 * noise[:, 2:]
        t = noise[:, 3]
    elif kind == "compression":             # shocked by div v, neighbours equal to 1e-9
        c[:, :2] *= 1.0 + 1e-9 * noise[:, :2]
        c[:, 1] *= 1e-6
        c[:, 2:] = -(x - x.mean(0))
        t = 1.0 + 1e-12 * noise[:, 0]
    elif kind == "tiny":                    # below the normal floats
        c[:, 0] = 1e-45 * (1 + 0.3 * noise[:, 0])
        c[:, 1] = 1e-45 * (1 + 0.3 * noise[:, 1])
        c[:, 2:] = 1e-42 * noise[:, 2:]
        t = 1e-50 * noise[:, 0]
    elif kind == "huge":                    # above them
        c[:, 0] = 1e40 * (1 + 0.3 * noise[:, 0])
        c[:, 1] = 1e45 * (1 + 0.3 * noise[:, 1])
        c[:, 2:] = 1e2 * noise[:, 2:]
        t = 1e60 * noise[:, 0]
    return c, t


KINDS = ("flat", "noise", "linear", "steps", "shocks", "compression", "tiny", "huge")


@pytest.mark.parametrize("which", sorted(MESHES))
@pytest.mark.parametrize("kind", KINDS)
def test_fluxes_and_tracer_slopes_equal_the_oracle(which, kind):
    mesh, ghost = MESHES[which]()
    cells, t = field(kind, mesh, np.random.default_rng(7))
    tr = np.stack([t, t[::-1], t * t], 1)
    stickers = np.zeros(mesh.n_cells, dtype=np.uint32)
    stickers[::17] = 1
    ev = np.zeros((mesh.n_faces, 2))
    for skip in (-1, 0):
        lp = oracle.lgi_params(ghost)
        ts = oracle.TracerSetup(3, limited=5, skip_sticker=skip, stickers=stickers)
        with richgpu.Handle(gamma=GAMMA, order=2, ghost_kind=ghost) as h:
            h.upload_mesh(mesh)
            h.set_tracer_config(3, limited=[0, 2], skip_sticker=skip, n_stickers=1)
            h.set_stickers(stickers)
            h.set_cells(cells)
            h.set_tracers(tr)
            h.set_edge_velocities(ev)
            try:
                want = oracle.flux_tr(mesh, cells, tr, ev, GAMMA, 2, lp, ts)
            except oracle.OracleError as err:
                # an unlimited neighbour (skip_key) can make a face state that
                # Hllc rejects: then both reject the same face
                with pytest.raises(richgpu.RichError) as got:
                    h.flux(0.0)
                assert (got.value.status, got.value.index) == (err.status, err.index)
                continue
            got = h.flux(0.0)
            slopes = h.tracer_slopes()
        assert np.array_equal(got, want[0])
        assert np.array_equal(slopes.reshape(-1), oracle.lgi_tr(mesh, cells, tr, GAMMA, lp, ts)[2].reshape(-1))


def test_random_mesh_reaches_cells_beyond_the_register_form():
    """8 neighbours are kept in registers: both forms of the kernel run above."""
    mesh, _ = MESHES["random"]()
    nn = np.diff(mesh.cell_face_offset)
    assert nn.max() > 8 and nn.min() <= 5 and abs(mesh.volume.sum() - 1.0) < 1e-12
