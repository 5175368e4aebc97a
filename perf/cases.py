"""The workloads whose speed this repository is held to.

A case is one pass of what a program does with a handle it keeps: load a state,
advance it through the public entry points (richgpu.Handle / Handle3, the C ABI
behind them), read the result back.  Host arrays are pinned, as a program that
streams state keeps them.  The listed cases cover the library's own workloads
(Sod and Sedov tubes and blasts, batches of Riemann problems, the adjoint, the
3D first-order path, the moving-mesh step, the plugin calls hdsim makes) from
the smallest mesh to the largest; draw() gives others of the same ranges.
exact() computes the same outputs in 64 bits with plain torch.
"""
import functools
import math
import os
import sys

import numpy as np
import torch
import torch.utils.checkpoint

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "huji-rich_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import richgpu  # noqa: E402
import synthetic  # noqa: E402
from meshview import FP32_MIXED, FP64  # noqa: E402

BOX = (-1.0, 1.0, -1.0, 1.0)
UNIT = (0.0, 1.0, 0.0, 1.0)


# ------------------------------------------------------------------ the cases

def listed():
    return [
        # the Sod tube at its own resolution: first order, FP64, 8,000 cells.
        # The smallest mesh in use; launches and latency decide it.
        {"name": "sod_200x40_fp64", "kind": "run", "nx": 200, "ny": 40, "mixed": False, "order": 1, "boundary": "rigid",
         "moving": False, "heun": False, "tracers": 0, "steps": 40},
        # the calls hdsim's plugins make on one moving-mesh step of a small
        # problem: upload, face velocities, dt, fluxes, extensives, cells
        {"name": "plugins_96x101_fp64", "kind": "plugins", "nx": 96, "ny": 101, "mixed": False, "order": 2,
         "boundary": "rigid"},
        # the headline problem on its bit-exact path, with face velocities
        {"name": "sedov_512_fp64", "kind": "run", "nx": 512, "ny": 512, "mixed": False, "order": 2, "boundary": "rigid",
         "moving": True, "heun": False, "tracers": 0, "steps": 10},
        # the headline problem and path: FP32-mixed, with face velocities
        {"name": "sedov_512_mixed", "kind": "run", "nx": 512, "ny": 512, "mixed": True, "order": 2, "boundary": "rigid",
         "moving": True, "heun": False, "tracers": 0, "steps": 40},
        # the largest mesh: beyond what the L2 cache holds, Eulerian
        {"name": "sedov_1024_mixed", "kind": "run", "nx": 1024, "ny": 1024, "mixed": True, "order": 2,
         "boundary": "rigid", "moving": False, "heun": False, "tracers": 0, "steps": 20},
        # TimeAdvance2Heun with tracers on a periodic box
        {"name": "periodic_256_heun_tracers_fp64", "kind": "run", "nx": 256, "ny": 256, "mixed": False, "order": 2,
         "boundary": "periodic", "moving": False, "heun": True, "tracers": 3, "steps": 5},
        # a batch of independent Riemann problems of uneven size, FP32-mixed,
        # replayed from a CUDA graph
        {"name": "riemann_batch_96_mixed", "kind": "batch", "problems": 96, "min_cells": 1024, "max_cells": 32768,
         "mixed": True, "steps": 20, "graph": True},
        # gradients of a 256 x 256 periodic run, FP64 and FP32-mixed: forward
        # with checkpoints, then the reverse sweep
        {"name": "adjoint_256_fp64", "kind": "adjoint", "nx": 256, "ny": 256, "mixed": False, "steps": 20, "every": 20},
        {"name": "adjoint_256_mixed", "kind": "adjoint", "nx": 256, "ny": 256, "mixed": True, "steps": 40, "every": 20},
        # the 3D first-order path at its own resolution
        {"name": "cube_96_fp64", "kind": "cube", "nx": 96, "ny": 96, "nz": 96, "mixed": False, "steps": 5},
        {"name": "cube_96_mixed", "kind": "cube", "nx": 96, "ny": 96, "nz": 96, "mixed": True, "steps": 20},
        # two moving-mesh steps end to end: motion, dt and fluxes on the
        # device, the next tessellation uploaded, state read back
        {"name": "moving_512_mixed", "kind": "moving", "nx": 512, "ny": 512, "mixed": True, "boundary": "rigid"},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _sides(rng, lo, hi):
    """An odd or even lattice, at most about 3 to 1."""
    nx = _log(rng, lo, hi)
    return nx, max(lo, min(hi, int(nx * math.exp(rng.uniform(-1.1, 1.1)))))


def draw(rng):
    kind = rng.choice(["run", "run", "run", "run", "batch", "adjoint", "cube", "moving", "plugins"])
    mixed = rng.random() < 0.5
    if kind == "run":
        heun = rng.random() < 0.2
        nx, ny = _sides(rng, 33, 512)
        return {"kind": kind, "nx": nx, "ny": ny, "mixed": mixed,
                "order": 2 if rng.random() < 0.8 else 1, "boundary": rng.choice(["rigid", "periodic"]),
                "moving": rng.random() < 0.5, "heun": heun,
                "tracers": rng.choice([0, 0, 0, 2, 5]) if not (mixed and heun) else 0, "steps": rng.randint(3, 10)}
    if kind == "batch":
        lo = _log(rng, 256, 2048)
        return {"kind": kind, "problems": _log(rng, 5, 64), "min_cells": lo, "max_cells": lo * rng.randint(2, 12),
                "mixed": mixed, "steps": rng.randint(3, 10), "graph": rng.random() < 0.5}
    if kind == "adjoint":
        nx, ny = _sides(rng, 33, 250)
        return {"kind": kind, "nx": nx, "ny": ny, "mixed": mixed,
                "steps": rng.randint(4, 16), "every": rng.randint(2, 10)}
    if kind == "cube":
        return {"kind": kind, "nx": rng.randint(17, 90), "ny": rng.randint(17, 90), "nz": rng.randint(17, 90),
                "mixed": mixed, "steps": rng.randint(2, 6)}
    nx, ny = _sides(rng, 33, 500 if kind == "moving" else 300)
    if kind == "moving":
        return {"kind": kind, "nx": nx, "ny": ny, "mixed": mixed, "boundary": rng.choice(["rigid", "periodic"])}
    return {"kind": kind, "nx": nx, "ny": ny, "mixed": mixed,
            "order": 2 if rng.random() < 0.8 else 1, "boundary": rng.choice(["rigid", "periodic"])}


# ------------------------------------------------------------------ inputs

@functools.lru_cache(maxsize=None)
def _lattice(nx, ny, box, boundary, seed, jitter):
    return synthetic.lattice_mesh(nx, ny, box, boundary, seed=seed, jitter=jitter)


@functools.lru_cache(maxsize=None)
def _batch(problems, lo, hi):
    """(mesh, offsets, gammas, cells) of a batch; the seeds of a case perturb its states."""
    mesh, offsets, gammas, cells, _ = synthetic.riemann_batch(problems, 11, lo, hi)
    return mesh, offsets, gammas, cells


@functools.lru_cache(maxsize=None)
def _cube(nx, ny, nz):
    return synthetic.cube_grid(nx, ny, nz, (-0.5, -0.5, -0.5), (0.5, 0.5, 0.5))


def _smooth(x, rng, amp, modes=6, period=2.0):
    """A seeded sum of Fourier modes at the points x (n, d), periodic over the box."""
    out = np.zeros(len(x))
    for _ in range(modes):
        k = rng.integers(-3, 4, x.shape[1])
        out += rng.normal(0, amp / math.sqrt(modes)) * np.sin(2 * np.pi / period * (x @ k) + rng.uniform(0, 2 * np.pi))
    return out


def _blast(mesh, rng, gamma):
    """A Sedov blast off the centre in a gas with smooth seeded density and velocity."""
    x = mesh.point_xy[:mesh.n_cells]
    c = np.zeros((mesh.n_cells, 4))
    c[:, 0] = 1.0 + _smooth(x, rng, 0.1)
    c[:, 1] = 1e-6
    centre = rng.uniform(-0.3, 0.3, 2)
    r = np.hypot(x[:, 0] - centre[0], x[:, 1] - centre[1])
    hot = r <= max(0.05, np.sort(r)[8])
    c[hot, 1] = (gamma - 1) / mesh.cd_volume[hot].sum()
    c[:, 2] = _smooth(x, rng, 0.02)
    c[:, 3] = _smooth(x, rng, 0.02)
    return c


def _waves(mesh, rng):
    """Smooth periodic flow: density, pressure and velocity from seeded modes."""
    x = mesh.point_xy[:mesh.n_cells]
    period = 1.0
    c = np.zeros((mesh.n_cells, 4))
    c[:, 0] = 1.0 + _smooth(x, rng, 0.1, period=period)
    c[:, 1] = 1.0 + _smooth(x, rng, 0.1, period=period)
    c[:, 2] = _smooth(x, rng, 0.2, period=period)
    c[:, 3] = _smooth(x, rng, 0.2, period=period)
    return c


def _tube(mesh, rng):
    """The Sod tube with seeded left and right states."""
    x = mesh.point_xy[:mesh.n_cells, 0]
    left = x < 0.5 * (x.min() + x.max())
    c = np.zeros((mesh.n_cells, 4))
    u = rng.uniform(0.9, 1.1, 4)
    c[:, 0] = np.where(left, 1.0 * u[0], 0.125 * u[1])
    c[:, 1] = np.where(left, 1.0 * u[2], 0.1 * u[3])
    return c


def _inputs(case, seed):
    """Everything of a case that does not depend on the library: mesh, gamma, state."""
    rng = np.random.default_rng([seed, 77])
    kind = case["kind"]
    if kind == "batch":
        mesh, offsets, gammas, cells = _batch(case["problems"], case["min_cells"], case["max_cells"])
        u = rng.uniform(0.8, 1.25, (len(gammas), 4))
        prob = np.repeat(np.arange(len(gammas)), np.diff(offsets))
        return {"mesh": mesh, "offsets": offsets, "gammas": gammas, "cells": cells * u[prob], "prob": prob,
                "gamma": gammas[prob]}
    if kind == "cube":
        n = (case["nx"], case["ny"], case["nz"])
        lo, hi = (-0.5, -0.5, -0.5), (0.5, 0.5, 0.5)
        x = synthetic.cube_centres(*n, lo, hi)
        cells = np.zeros((len(x), 5))
        cells[:, 0] = 1.0 + _smooth(x, rng, 0.1)
        r = np.sqrt(((x - rng.uniform(-0.2, 0.2, 3)) ** 2).sum(1))
        cells[:, 1] = np.where(r < 0.08, 100.0, 1e-3)
        for k in range(3):
            cells[:, 2 + k] = _smooth(x, rng, 0.05)
        return {"mesh": _cube(*n), "cells": cells, "gamma": 5.0 / 3.0}
    if kind == "adjoint":
        mesh = _lattice(case["nx"], case["ny"], UNIT, "periodic", 9, 1e-3)
        cells = _waves(mesh, rng)
        width = np.sqrt(mesh.volume.min() / np.pi)
        dt = 0.3 * width / 2.5
        return {"mesh": mesh, "cells": cells, "gamma": 5.0 / 3.0, "dt": dt,
                "bar": rng.normal(0, 1.0, (mesh.n_cells, 4)) * mesh.cd_volume[:, None]}
    gamma = 5.0 / 3.0
    periodic = case["boundary"] == "periodic"
    box = UNIT if periodic else BOX
    jitter = 0.05 if kind in ("moving", "plugins") else 1e-3
    if case.get("order", 2) == 1 and not periodic:
        gamma, box = 1.4, (0.0, 1.0, 0.0, case["ny"] / case["nx"])
    mesh = _lattice(case["nx"], case["ny"], box, case["boundary"], 2, jitter)
    if periodic:
        cells = _waves(mesh, rng)
    elif case.get("order", 2) == 1:
        cells = _tube(mesh, rng)
    else:
        cells = _blast(mesh, rng, gamma)
    got = {"mesh": mesh, "cells": cells, "gamma": gamma, "box": box}
    x = mesh.point_xy[:mesh.n_cells]
    period = box[1] - box[0]
    if kind == "moving":
        got["mesh2"] = _lattice(case["nx"], case["ny"], box, case["boundary"], 3, jitter)
    if case.get("moving") or kind == "plugins":
        pv = np.stack([_smooth(x, rng, 0.05, period=period), _smooth(x, rng, 0.05, period=period)], 1)
        got["ev"] = synthetic.face_velocities(mesh, pv)
    if case.get("tracers"):
        got["tracers"] = np.stack([1.0 + _smooth(x, rng, 0.2, period=period) for _ in range(case["tracers"])], 1)
    return got


def _pin(a):
    t = torch.empty(a.shape, dtype=torch.float64, pin_memory=True)
    t.numpy()[...] = a
    return t.numpy()


def _pinned(*shape):
    return torch.empty(shape, dtype=torch.float64, pin_memory=True).numpy()


def _pin_mesh(mesh):
    """The mesh's arrays in pinned host memory (what a program that uploads every step keeps)."""
    arrays = {}
    for k in ("point_xy", "cm_xy", "volume", "cd_volume", "ghost_source", "ghost_face", "face_cells", "face_vertices",
              "cell_face_offset", "cell_faces"):
        a = getattr(mesh, k)
        t = torch.empty(a.shape, dtype=torch.from_numpy(a).dtype, pin_memory=True)
        t.numpy()[...] = a
        arrays[k] = t.numpy()
    return type(mesh)(**arrays)


def _extensives(mesh, c, gamma):
    m = mesh.cd_volume * c[:, 0]
    e = c[:, 1] / c[:, 0] / (gamma - 1) * m + 0.5 * m * (c[:, 2] ** 2 + c[:, 3] ** 2)
    return np.stack([m, e, c[:, 2] * m, c[:, 3] * m], 1)


def prepare(case, seed):
    d = _inputs(case, seed)
    kind, mesh = case["kind"], d["mesh"]
    precision = FP32_MIXED if case["mixed"] else FP64
    n = mesh.n_cells
    s = {"case": case}
    if kind == "cube":
        h = richgpu.Handle3(gamma=d["gamma"], precision=precision)
        h.upload_mesh(mesh)
        c = d["cells"]
        vol = mesh.volume[:, None]
        en = c[:, :1] * (0.5 * (c[:, 2:] ** 2).sum(1, keepdims=True) + c[:, 1:2] / c[:, :1] / (d["gamma"] - 1))
        s.update(h=h, cells=_pin(c), ext=_pin(np.concatenate([vol * c[:, :1], c[:, :1] * c[:, 2:] * vol, vol * en], 1)))
        return s
    periodic = kind == "adjoint" or case.get("boundary") == "periodic"
    kw = {"gamma": 1.4 if kind == "batch" else d["gamma"], "order": case.get("order", 2),
          "ghost_kind": 1 if periodic else 0, "precision": precision}
    if case.get("heun"):
        kw["time_integrator"] = 1
    h = richgpu.Handle(**kw)
    s.update(h=h, cells=_pin(d["cells"]), out=(_pinned(n, 4), _pinned(n, 4)))
    if kind == "adjoint":
        h.upload_mesh(mesh)
        s.update(dt=d["dt"], bar=_pin(d["bar"]))
        return s
    s["ext"] = _pin(_extensives(mesh, d["cells"], d["gamma"]))
    if kind == "moving":
        b = d["box"]
        h.set_outer_box(*b)
        h.set_point_motion(kind=2, edges=1 if periodic else 0)
        s["meshes"] = (_pin_mesh(mesh), _pin_mesh(d["mesh2"]))
        s["pv"] = (_pinned(n, 2), _pinned(n, 2))
        h.upload_mesh(s["meshes"][0], richgpu.MESH_DEVICE_GEOMETRY)
        return s
    if kind == "plugins":
        s.update(mesh=_pin_mesh(mesh), ev=_pin(d["ev"]))
        h.upload_mesh(s["mesh"])
        return s
    if case.get("tracers"):
        h.set_tracer_config(case["tracers"], limited=tuple(range(0, case["tracers"], 2)))
    h.upload_mesh(mesh)
    if kind == "batch":
        h.set_problems(d["offsets"], d["gammas"])
    h.set_edge_velocities(d["ev"] if "ev" in d else np.zeros((mesh.n_faces, 2)))
    if case.get("tracers"):
        s["tracers"] = _pin(d["tracers"])
        s["tracer_ext"] = _pin(d["tracers"] * (mesh.cd_volume * d["cells"][:, 0])[:, None])
    return s


# ------------------------------------------------------------------ one pass

def run(s):
    case, h = s["case"], s["h"]
    kind = case["kind"]
    if kind == "cube":
        h.set_cells(s["cells"])
        h.set_extensives(s["ext"])
        dts = h.run(case["steps"])
        return {"cells": h.get_cells(), "ext": h.get_extensives(), "dt": dts}
    cells, ext = s["out"]
    if kind == "adjoint":
        h.set_cells(s["cells"])
        h.step_fwd(case["steps"], s["dt"], case["every"])
        grad = h.step_bwd(s["bar"])
        return {"cells": h.get_cells(cells), "grad": grad}
    h.set_cells(s["cells"])
    h.set_extensives(s["ext"])
    if kind == "moving":
        a, b = s["meshes"]
        dt0, pv0 = h.advance_begin(out=s["pv"][0])
        h.upload_mesh(b, richgpu.MESH_DEVICE_GEOMETRY)
        h.cell_update()
        dt1, pv1 = h.advance_begin(out=s["pv"][1])
        h.upload_mesh(a, richgpu.MESH_DEVICE_GEOMETRY)
        h.cell_update()
        h.get_state_async(cells, ext)
        h.wait_state()
        return {"cells": cells, "ext": ext, "dt": [dt0, dt1], "pv": [pv0, pv1]}
    if kind == "plugins":
        h.upload_mesh(s["mesh"])
        h.set_edge_velocities(s["ev"])
        dt = h.cfl_dt()
        fluxes = h.flux(dt)
        h.extensive_update(dt)
        h.cell_update()
        return {"cells": h.get_cells(cells), "ext": h.get_extensives(ext), "dt": dt, "fluxes": fluxes}
    if case.get("tracers"):
        h.set_tracers(s["tracers"])
        h.set_extensive_tracers(s["tracer_ext"])
    if kind == "batch":
        # a batch's results: the states and each problem's last dt
        if case["graph"]:
            h.run_graph(case["steps"])
        else:
            h.run(case["steps"])
        return {"cells": h.get_cells(cells), "ext": h.get_extensives(ext), "dt": h.problem_times()[1]}
    got = {"dt": h.run(case["steps"]), "cells": h.get_cells(cells), "ext": h.get_extensives(ext)}
    if case.get("tracers"):
        got["tracers"] = h.get_tracers()
        got["tracer_ext"] = h.get_extensive_tracers()
    return got


def _counts(case):
    if case["kind"] == "batch":
        n = sum(synthetic.riemann_problem_cells(p, 11, case["min_cells"], case["max_cells"])
                for p in range(case["problems"]))
        return n, 3 * n
    if case["kind"] == "cube":
        n = case["nx"] * case["ny"] * case["nz"]
        return n, 3 * n
    n = case["nx"] * case["ny"]
    return n, 3 * n


def work(case):
    """Per step: the state (cells and extensives) read and written once, each
    face's topology and geometry read once; the arithmetic of the
    reconstruction, the Riemann solver and the update."""
    n, e = _counts(case)
    kind, cell = case["kind"], 16 if case["mixed"] else 32
    real = 4 if case["mixed"] else 8
    steps = case.get("steps", 2 if kind == "moving" else 1)
    if kind == "cube":
        return {"bytes": steps * (n * 2 * (48 + 5 * real) + e * (8 + 4 * real)), "flops": steps * (n * 60.0 + e * 220.0)}
    per_step = n * 2 * (32 + cell) + e * (8 + 8 * real)
    flops = n * 60.0 + e * 200.0
    if case.get("order", 2) == 2:
        flops += n * 400.0
    k = case.get("tracers", 0)
    per_step += n * k * 32
    flops += (n * 80.0 + e * 8.0) * k
    if case.get("heun"):
        per_step, flops = 2 * per_step, 2 * flops
    if kind == "adjoint":
        # forward, the recomputed forward and the reverse sweep of each step
        per_step, flops = 3 * per_step, 4 * flops
    if kind in ("moving", "plugins"):
        # the mesh itself: points, topology, vertices
        per_step += n * (16 + 4 + 24) + e * 40
    return {"bytes": float(steps * per_step), "flops": float(steps * flops)}


# ------------------------------------------------------------------ 64 bits

class _Mesh:
    """A packed 2D mesh as torch tensors, each cell's faces padded to one width."""

    def __init__(self, m, order, dev, periodic):
        def t(a):
            return torch.from_numpy(np.ascontiguousarray(a)).to(dev)
        n = self.n = m.n_cells
        self.periodic, self.order = periodic, order
        self.x, self.cm, self.vol, self.cdv = t(m.point_xy), t(m.cm_xy), t(m.volume), t(m.cd_volume)
        src = np.concatenate([np.arange(n), m.ghost_source.astype(np.int64)])
        fc = m.face_cells.astype(np.int64)
        self.src, self.fc, self.fv = t(src), t(fc), t(m.face_vertices)
        # the cell a ghost's state is formed from: the real side of its face
        real = m.ghost_source.astype(np.int64).copy()
        if not periodic:
            gf = m.ghost_face
            has = gf >= 0
            f = fc[gf[has]]
            real[has] = np.where(f[:, 0] >= n, f[:, 1], f[:, 0])
            g0, g1 = m.point_xy[f[:, 0]], m.point_xy[f[:, 1]]
            nr = np.where((f[:, 0] >= n)[:, None], g0 - g1, g1 - g0)
            unit = np.zeros((m.n_ghosts, 2))
            unit[has] = nr / np.hypot(nr[:, 0], nr[:, 1])[:, None]
            self.unit = t(unit)
        self.real = t(real)
        off = m.cell_face_offset.astype(np.int64)
        cnt = np.diff(off)
        k = int(cnt.max())
        slot = off[:-1, None] + np.arange(k)[None]
        mask = np.arange(k)[None] < cnt[:, None]
        face = m.cell_faces.astype(np.int64)[np.where(mask, slot, 0)]
        first = fc[face, 0] == np.arange(n)[:, None]
        other = np.where(first, fc[face, 1], fc[face, 0])
        other = np.where(mask, other, 0)
        self.mask, self.face, self.other = t(mask), t(face), t(other)
        self.sign = t(np.where(mask, np.where(first, -1.0, 1.0), 0.0))
        # face geometry
        v0, v1 = self.fv[:, :2], self.fv[:, 2:]
        self.par = v1 - v0
        self.area = self.par.norm(dim=1)
        mid = 0.5 * (v0 + v1)
        a, b = self.fc[:, 0], self.fc[:, 1]
        if order == 1:
            self.nrm = self.x[b] - self.x[a]
        else:
            w = torch.where((a < n)[:, None], v0 - self.x[a], self.x[b] - v0)
            self.nrm = w - self.par * ((w * self.par).sum(1) / (self.par ** 2).sum(1))[:, None]
        self.nabs = self.nrm.norm(dim=1)
        self.dm = (mid - self.cm[a], mid - self.cm[b])
        self.width = torch.sqrt(self.vol / math.pi)
        self.mirror_face = self.src[a] == self.src[b]
        mirror = self.mirror_face[self.face] & self.mask
        self.mirror = mirror
        self.boundary = mirror.any(1)
        if order == 2:
            i = torch.arange(n, device=dev)[:, None]
            mk = self.mask[..., None].double()
            d = self.x[self.other] - self.x[:n, None]
            r = d / torch.where(self.mask[..., None], d, torch.ones_like(d)).norm(dim=2, keepdim=True)
            r = r * self.area[self.face][..., None] * mk
            c = mid[self.face] - 0.5 * (self.cm[self.other] + self.cm[:n, None])
            eye = torch.eye(2, dtype=torch.float64, device=dev)
            mat = self.vol[:, None, None] * eye - torch.einsum("nkr,nkc->nrc", r, c)
            self.h = torch.where(self.boundary[:, None, None], (self.cm[self.other] - self.cm[:n, None]) * mk, 0.5 * r)
            hb = self.h
            sq = torch.einsum("nkr,nkc->nrc", hb, hb)
            self.inv = torch.linalg.inv(torch.where(self.boundary[:, None, None], sq, mat))
            self.cdm = mid[self.face] - self.cm[i]  # centroid - CM of the cell, per entry

    def points(self, w):
        """States of all points, the ghosts' formed from their cells."""
        g = w[self.real]
        if not self.periodic and len(g):
            s = 2 * (g[:, 2] * self.unit[:, 0] + g[:, 3] * self.unit[:, 1])
            g = torch.cat([g[:, :2], g[:, 2:4] - self.unit * s[:, None], g[:, 4:]], 1)
        return torch.cat([w, g], 0)

    def slopes(self, w, p, gamma, limited):
        """LinearGaussImproved slopes (n, q, 2) of cell states w (n, q): the four
        hydro fields, then tracers; limited: which tracers keep a slope."""
        nb = p[self.other]
        mask = self.mask[..., None]
        cell = w[:, None]
        base = torch.where(self.boundary[:, None, None], nb - cell, nb + cell)
        v = torch.einsum("nkq,nkr->nqr", base * mask, self.h)
        s = torch.einsum("nrc,nqc->nqr", self.inv, v)
        if limited is not None:
            s = s * limited[None, :, None]
        ratio = torch.minimum(nb[..., 1], cell[..., 1]) / torch.maximum(nb[..., 1], cell[..., 1])
        cs = torch.sqrt(gamma * w[:, 1] / w[:, 0])
        shock = (((s[:, 2, 0] + s[:, 3, 1]) * self.width < -0.2 * cs) | ((ratio < 0.7) & self.mask).any(1))
        shock = shock[:, None]
        count = mask & (shock[..., None] | ~self.mirror[..., None])
        hi = torch.where(count, nb, cell).amax(1)
        lo = torch.where(count, nb, cell).amin(1)
        hi, lo = torch.maximum(hi, w), torch.minimum(lo, w)
        up, down = hi - w, lo - w
        thr = torch.where(shock, 0.1, 0.05) * torch.maximum(up.abs(), down.abs())
        dphi = torch.einsum("nkr,nqr->nkq", self.cdm, s)
        cv = cell + dphi
        active = mask & ((dphi.abs() > thr[:, None]) | (cv * cell < 0))
        t = 1e-9 * cell
        vel = torch.arange(w.shape[1], device=w.device) >= 2
        ta = torch.where(vel, t.abs(), t)
        rise, fall = dphi > ta, dphi < -ta
        plain = active & (rise | fall)
        dead = torch.where(torch.arange(w.shape[1], device=w.device) >= 4, t.abs(), t)
        shocked = active & (dphi.abs() > dead)
        use = torch.where(shock[..., None], shocked, plain)
        num = torch.where(shock[..., None], 0.5 * (nb - cell), torch.where(rise, up[:, None], down[:, None]))
        cand = torch.where(use, num, 1.0) / torch.where(use, dphi, 1.0)
        cand = torch.where(shock[..., None], cand.clamp(min=0.0), cand)
        psi = torch.minimum(cand.amin(1), torch.ones_like(w))
        return s * psi[..., None]

    def dt(self, w, ev, gamma, prob, n_prob):
        cs = torch.sqrt(gamma * w[:, 1] / w[:, 0])
        rel = (w[:, None, 2:4] - ev[self.face]).norm(dim=2)
        rel = torch.where(self.mask, rel, 0.0).amax(1)
        bound = self.width / (cs + rel)
        if prob is None:
            return 0.3 * bound.min()
        return 0.3 * torch.full((n_prob,), math.inf, dtype=w.dtype, device=w.device).scatter_reduce(0, prob, bound, "amin")

    def fluxes(self, w, ev, gamma, limited=None):
        """Per face {mass, energy, px, py, tracers...}, unscaled."""
        a, b = self.fc[:, 0], self.fc[:, 1]
        n = self.n
        real = torch.where(a < n, a, b)
        g = gamma[real]
        if self.order == 2:
            p = self.points(w)
            s = self.slopes(w, p, gamma, limited)
            side = []
            for pid, dm in ((a, self.dm[0]), (b, self.dm[1])):
                grad = s[self.src[pid]]
                if not self.periodic:
                    grad = grad * (pid < n)[:, None, None]
                side.append(p[pid] + torch.einsum("eqr,er->eq", grad, dm))
            l, r = side
        else:
            l, r = w[self.src[a]], w[self.src[b]]
            axis = self.par / self.area[:, None]

            def mirrored(q):
                v = 2 * (q[:, 2:4] * axis).sum(1, keepdim=True) * axis - q[:, 2:4]
                return torch.cat([q[:, :2], v, q[:, 4:]], 1)
            m = self.mirror_face
            l, r = (torch.where((m & (a >= n))[:, None], mirrored(r), l), torch.where((m & (b >= n))[:, None], mirrored(l), r))
        nn, pp = self.nrm / self.nabs[:, None], self.par / self.area[:, None]
        vel = (nn * ev).sum(1)

        def frame(q):
            return [q[:, 0], q[:, 1], (q[:, 2:4] * nn).sum(1) - vel, (q[:, 2:4] * pp).sum(1)]
        m, mx, my, en = _hllc(frame(l), frame(r), g)
        en = en + mx * vel + 0.5 * m * vel * vel
        mx = mx + vel * m
        mom = nn * mx[:, None] + pp * my[:, None]
        out = torch.cat([m[:, None], en[:, None], mom], 1)
        if w.shape[1] > 4:
            t = torch.where((m > 0)[:, None], l[:, 4:], r[:, 4:])
            if self.order == 1:
                up_ghost = torch.where(m > 0, a, b) >= n
                t = t * ~(self.mirror_face & up_ghost)[:, None]
            out = torch.cat([out, m[:, None] * t], 1)
        return out

    def gather(self, f):
        return (f[self.face] * self.sign[..., None]).sum(1)

    def cells(self, u, gamma, cdv):
        d, v = u[:, 0] / cdv, u[:, 2:4] / u[:, :1]
        e = u[:, 1] / u[:, 0] - 0.5 * (v ** 2).sum(1)
        return torch.cat([d[:, None], ((gamma - 1) * e * d)[:, None], v, u[:, 4:] / u[:, :1]], 1)


def _hllc(l, r, g):
    dl, pl, ul, tl = l
    dr, pr, ur, tr = r
    cl, cr = torch.sqrt(g * pl / dl), torch.sqrt(g * pr / dr)
    sl, sr = torch.minimum(ul - cl, ur - cr), torch.maximum(ul + cl, ur + cr)
    ss = (pr - pl + dl * ul * (sl - ul) - dr * ur * (sr - ur)) / (dl * (sl - ul) - dr * (sr - ur))
    left = (sl > 0) | ((sl <= 0) & (ss >= 0))
    d, p, u, t = (torch.where(left, x, y) for x, y in zip(l, r))
    sk = torch.where(left, sl, sr)
    ek = 0.5 * d * (u * u + t * t) + p / (g - 1)
    m, mx, my, en = d * u, p + d * u * u, d * u * t, (ek + p) * u
    star = torch.where(left, ~(sl > 0), ~(sr < 0))
    ds = d * (sk - u) / (sk - ss)
    use = ek * ds / d + ds * (ss - u) * (ss + p / (d * (sk - u)))
    z = torch.zeros_like(m)
    return (m + torch.where(star, sk * (ds - d), z), mx + torch.where(star, sk * (ds * ss - d * u), z),
            my + torch.where(star, sk * (ds * t - d * t), z), en + torch.where(star, sk * (use - ek), z))


def _exact_run(case, d, dev):
    periodic = case.get("boundary") == "periodic"
    m = _Mesh(d["mesh"], case.get("order", 2), dev, periodic)

    def t(a):
        return torch.from_numpy(np.ascontiguousarray(a)).to(dev)
    w = t(d["cells"])
    gamma = t(np.broadcast_to(np.asarray(d["gamma"], dtype=np.float64), (m.n,)).copy())
    u = t(_extensives(d["mesh"], d["cells"], d["gamma"]))
    ev = t(d["ev"]) if "ev" in d else torch.zeros(len(m.fc), 2, dtype=torch.float64, device=dev)
    limited = None
    k = case.get("tracers", 0)
    if k:
        w = torch.cat([w, t(d["tracers"])], 1)
        u = torch.cat([u, t(d["tracers"]) * u[:, :1]], 1)
        limited = torch.ones(4 + k, dtype=torch.float64, device=dev)
        limited[5::2] = 0.0
    prob, n_prob, fp = None, 0, None
    if "prob" in d:
        prob, n_prob = t(d["prob"].astype(np.int64)), len(d["gammas"])
        fp = prob[m.src[m.fc[:, 0]]]
    dts = []
    for _ in range(case.get("steps", 1)):
        dt = m.dt(w, ev, gamma, prob, n_prob)
        scale = ((dt if prob is None else dt[fp]) * m.area)[:, None]
        f = m.fluxes(w, ev, gamma, limited)
        new = u + m.gather(f * scale)
        if case.get("heun"):
            mid = m.cells(new, gamma, m.cdv)
            new = 0.5 * (new + m.gather(m.fluxes(mid, ev, gamma, limited) * scale) + u)
        u, w = new, m.cells(new, gamma, m.cdv)
        dts.append(dt)
    got = {"cells": w[:, :4], "ext": u[:, :4], "dt": dts[-1] if prob is not None else torch.stack(dts)}
    if k:
        got["tracers"], got["tracer_ext"] = w[:, 4:], u[:, 4:]
    if case["kind"] == "plugins":
        got["dt"], got["fluxes"] = dts[0], f
    return got


def _exact_moving(case, d, dev):
    periodic = case["boundary"] == "periodic"
    a, b = (_Mesh(x, 2, dev, periodic) for x in (d["mesh"], d["mesh2"]))
    w = torch.from_numpy(d["cells"]).to(dev)
    u = torch.from_numpy(_extensives(d["mesh"], d["cells"], d["gamma"])).to(dev)
    gamma = torch.full((a.n,), d["gamma"], dtype=torch.float64, device=dev)
    got = {"dt": [], "pv": []}
    for m, after in ((a, b), (b, a)):
        r = m.cm[:m.n] - m.x[:m.n]
        cs = torch.maximum(torch.sqrt(gamma * w[:, 1] / w[:, 0]), w[:, 2:4].norm(dim=1))
        move = r * (0.15 * cs / m.width)[:, None]
        pv = w[:, 2:4] + torch.where((r.norm(dim=1) < 0.9 * 0.02 * m.width)[:, None], 0.0, move)
        fa, fb = m.fc[:, 0], m.fc[:, 1]
        wl, wr = pv[m.src[fa]], pv[m.src[fb]]
        dx = m.x[fb] - m.x[fa]
        off = 0.5 * (m.fv[:, :2] + m.fv[:, 2:]) - 0.5 * (m.x[fa] + m.x[fb])
        ev = 0.5 * (wl + wr) + dx * (((wl - wr) * off).sum(1) / (dx * dx).sum(1))[:, None]
        if not periodic:
            ev = torch.where(m.mirror_face[:, None], 0.0, ev)
        dt = m.dt(w, ev, gamma, None, 0)
        u = u + m.gather(m.fluxes(w, ev, gamma) * (dt * m.area)[:, None])
        w = m.cells(u, gamma, after.cdv)
        got["dt"].append(dt)
        got["pv"].append(pv)
    return {"cells": w, "ext": u, **got}


def _exact_adjoint(case, d, dev):
    m = _Mesh(d["mesh"], 2, dev, True)
    gamma = torch.full((m.n,), d["gamma"], dtype=torch.float64, device=dev)
    ev = torch.zeros(len(m.fc), 2, dtype=torch.float64, device=dev)
    scale = (d["dt"] * m.area)[:, None]
    w0 = torch.from_numpy(d["cells"]).to(dev).requires_grad_(True)

    def start(w):
        mass = m.cdv * w[:, 0]
        return torch.stack([mass, w[:, 1] / (d["gamma"] - 1) * m.cdv + 0.5 * mass * (w[:, 2] ** 2 + w[:, 3] ** 2),
                            mass * w[:, 2], mass * w[:, 3]], 1)

    def step(u, w):
        u = u + m.gather(m.fluxes(w, ev, gamma) * scale)
        return u, m.cells(u, gamma, m.cdv)
    u, w = start(w0), w0
    for _ in range(case["steps"]):
        u, w = torch.utils.checkpoint.checkpoint(step, u, w, use_reentrant=False)
    (w * torch.from_numpy(d["bar"]).to(dev)).sum().backward()
    return {"cells": w.detach(), "grad": w0.grad}


def _exact_cube(case, d, dev):
    m = d["mesh"]

    def t(a):
        return torch.from_numpy(np.ascontiguousarray(a)).to(dev)
    fc = t(m.face_cells.astype(np.int64))
    a, b = fc[:, 0], fc[:, 1]
    n = t(m.face_normal)
    n = n / n.norm(dim=1, keepdim=True)
    area, vol, width = t(m.face_area), t(m.volume), t(m.width)
    g = d["gamma"]
    w = t(d["cells"])
    u = torch.cat([w[:, :1], w[:, :1] * w[:, 2:],
                   w[:, :1] * 0.5 * (w[:, 2:] ** 2).sum(1, keepdim=True) + w[:, 1:2] / (g - 1)], 1) * vol[:, None]
    wall = (a < 0) | (b < 0)
    ia, ib = torch.where(a < 0, b, a), torch.where(b < 0, a, b)
    dts = []
    for _ in range(case["steps"]):
        dt = 0.3 * (width / (w[:, 2:].norm(dim=1) + torch.sqrt(g * w[:, 1] / w[:, 0]))).min()
        wa, wb = w[ia], w[ib]

        def reflected(q, c):
            v = q[:, 2:] - 2 * (q[:, 2:] * n).sum(1, keepdim=True) * n
            return torch.where(c[:, None], torch.cat([q[:, :2], v], 1), q)
        wa, wb = reflected(wa, a < 0), reflected(wb, b < 0)

        def prim(q):
            vn = (q[:, 2:] * n).sum(1)
            return [q[:, 0], q[:, 1], vn, (q[:, 2:] - vn[:, None] * n).norm(dim=1)]
        mass, mx, my, en = _hllc(prim(wa), prim(wb), torch.tensor(g, dtype=torch.float64, device=dev))
        donor = torch.where((mass > 0)[:, None], wa[:, 2:], wb[:, 2:])
        donor = torch.where(wall[:, None], torch.where((a < 0)[:, None], wb[:, 2:], wa[:, 2:]), donor)
        par = donor - (donor * n).sum(1, keepdim=True) * n
        p, v = par.norm(dim=1, keepdim=True), donor.norm(dim=1, keepdim=True)
        par = torch.where(v < 1e-9, par, par / torch.where(v < 1e-9, 1.0, torch.where(p < 1e-8 * v, v, p)))
        f = torch.cat([mass[:, None], mx[:, None] * n + my[:, None] * par, en[:, None]], 1) * (dt * area)[:, None]
        u = u.index_add(0, ia[a >= 0], -f[a >= 0]).index_add(0, ib[b >= 0], f[b >= 0])
        vel = u[:, 1:4] / u[:, :1]
        dens = u[:, 0] / vol
        e = u[:, 4] / u[:, 0] - 0.5 * (vel ** 2).sum(1)
        w = torch.cat([dens[:, None], ((g - 1) * e * dens)[:, None], vel], 1)
        dts.append(dt)
    return {"cells": w, "ext": u, "dt": torch.stack(dts)}


def exact(case, seed):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    d = _inputs(case, seed)
    kind = case["kind"]
    if kind == "cube":
        return _exact_cube(case, d, dev)
    if kind == "adjoint":
        return _exact_adjoint(case, d, dev)
    if kind == "moving":
        return _exact_moving(case, d, dev)
    return _exact_run(case, d, dev)
