"""The reverse of one face (rg_adjoint_rev.cu) where its branches differ: flow
supersonic either way (an undisturbed side), at rest (zeros in most products),
wave speeds taken from the other side or crossed.

Dot-product test <Wbar, TLM dW> = <ADJ Wbar, dW>: each side is the result of
about 1,000 dependent roundings per step over 3 steps, a condition of 10 at
most, so the two agree within 1e-11 of the sums of magnitudes.
"""
import numpy as np
import pytest

import richgpu
import synthetic

pytestmark = pytest.mark.gpu

GAMMA = 5 / 3


def flow(mesh, kind, rng):
    n = mesh.n_cells
    c = np.empty((n, 4))
    c[:, 0] = np.exp(rng.normal(0, 0.3, n))
    c[:, 1] = np.exp(rng.normal(0, 0.3, n))
    c[:, 2:] = rng.normal(0, 0.2, (n, 2))
    if kind == "right":
        c[:, 2] += 5.0
    elif kind == "left":
        c[:, 2] -= 5.0
    elif kind == "down":
        c[:, 3] -= 5.0
    elif kind == "rest":
        c[:, 2:] = 0.0
    elif kind == "clash":  # neighbours at Mach 3 towards and away from each other
        c[:, 2:] = rng.choice([-4.0, 4.0], (n, 2))
    elif kind == "contrast":  # sound speeds 100 to 1: both waves of a face from one side
        c[:, 1] = np.where(rng.random(n) < 0.5, 1e4, 1.0)
    return c


@pytest.mark.parametrize("nx,ny", [(7, 9), (33, 21)])
@pytest.mark.parametrize("kind", ["right", "left", "down", "rest", "clash", "contrast"])
def test_dot_product(kind, nx, ny):
    mesh = synthetic.lattice_mesh(nx, ny, (0.0, 1.0, 0.0, 1.0), "periodic", seed=5)
    rng = np.random.default_rng(nx)
    cells = flow(mesh, kind, rng)
    wbar, dw = rng.normal(size=cells.shape), rng.normal(size=cells.shape)
    with richgpu.Handle(gamma=GAMMA, order=2, ghost_kind=1, device=0) as h:
        h.upload_mesh(mesh)
        h.set_edge_velocities(np.zeros((mesh.n_faces, 2)))
        h.set_cells(cells)
        dt = 0.1 * h.cfl_dt()
        h.step_fwd(3, dt, 2)
        g = h.step_bwd(wbar)
        h.set_cells(cells)
        tl = h.step_tlm(3, dt, dw)
    lhs, rhs = float(np.sum(wbar * tl)), float(np.sum(g * dw))
    scale = float(np.sum(np.abs(wbar * tl)) + np.sum(np.abs(g * dw)))
    assert abs(lhs - rhs) <= 1e-11 * scale, (lhs, rhs, scale)
