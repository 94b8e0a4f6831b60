"""Performance cases of the lattice Boltzmann library: what a user's program asks of it.

Every case is a set-up that the repository itself runs (the cavities, channel, porous medium,
Taylor-Green box and request mix of its examples, tests and benchmark, at their sizes or at
generic ones) and one pass is what such a program repeats: a number of time steps, and what it
reads in between.  Outputs are the populations themselves, as views of the lattice's device
columns (`population_ptr`), or the fields that the program reads.

listed() names the cases, draw(rng) makes further ones of the same ranges, prepare() builds the
lattice, run() makes a pass, work() counts what a pass cannot do without, and exact() computes
the same outputs in 64 bits with plain torch.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from openlb_b200 import configs, lbx

# Velocities c_i and weights of the descriptors, in the order the populations are exchanged in.
_C9 = [(0, 0, 0), (-1, 1, 0), (-1, 0, 0), (-1, -1, 0), (0, -1, 0), (1, -1, 0), (1, 0, 0), (1, 1, 0), (0, 1, 0)]
_H19 = [(-1, 0, 0), (0, -1, 0), (0, 0, -1), (-1, -1, 0), (-1, 1, 0), (-1, 0, -1), (-1, 0, 1), (0, -1, -1), (0, -1, 1)]
_H27 = _H19 + [(-1, -1, -1), (-1, -1, 1), (-1, 1, -1), (-1, 1, 1)]


def _both(half):
    return [(0, 0, 0)] + half + [tuple(-v for v in c) for c in half]


_C = {9: _C9, 19: _both(_H19), 27: _both(_H27)}
_W = {9: {0: 4 / 9, 1: 1 / 9, 2: 1 / 36},
      19: {0: 1 / 3, 1: 1 / 18, 2: 1 / 36},
      27: {0: 8 / 27, 1: 2 / 27, 2: 1 / 54, 3: 1 / 216}}
_BYTES = {"f64": 8, "f32": 4, "f16dev": 2}
_TYPE = {"f64": "<f8", "f32": "<f4", "f16dev": "<f2"}
# Floating-point operations of one cell's collision: the moments, q equilibria and relaxations,
# and what the model adds (a plain count of the formulas; the traffic bounds every case).
_FLOPS = {"bgk": 13, "trt": 18, "smagorinsky_forced_bgk": 30}


def _weight(q, c):
    return _W[q][sum(abs(v) for v in c)]


def listed():
    return [
        # The smallest call: the 2D lid-driven cavity of the C++ example (interpolated velocity
        # walls and lid, FP64) at the size of the 20,000-step accuracy run; latency and launches.
        {"name": "cavity2d_128", "kind": "cavity2d", "nx": 128, "ny": 128, "storage": "f64", "steps": 100},
        # A larger 2D cavity with halfway bounce-back walls and a moving lid, FP32, odd extents.
        {"name": "cavity2d_1001", "kind": "links", "q": 9, "nx": 1001, "ny": 999, "nz": 1, "storage": "f32",
         "steps": 50},
        # The 3D lid-driven cavity as a single solve: 100 steps, then the convergence residual.
        {"name": "cavity3d_64", "kind": "links", "q": 19, "nx": 64, "ny": 64, "nz": 64, "storage": "f32",
         "steps": 100},
        # A box watched closely: every step with statistics that the host reads.
        {"name": "monitor_96", "kind": "monitor", "q": 19, "nx": 96, "ny": 96, "nz": 96, "dynamics": "bgk",
         "storage": "f32", "steps": 20, "tuned": False},
        # The benchmark's Taylor-Green box, FP32 and in the 16-bit storage form, autotuned as there.
        {"name": "box_256_f32", "kind": "box", "q": 19, "nx": 256, "ny": 256, "nz": 256, "dynamics": "bgk",
         "storage": "f32", "steps": 20, "tuned": True},
        {"name": "box_256_f16", "kind": "box", "q": 19, "nx": 256, "ny": 256, "nz": 256, "dynamics": "bgk",
         "storage": "f16dev", "steps": 20, "tuned": True},
        # A ragged FP64 box with the default launch shape.
        {"name": "box_ragged_f64", "kind": "box", "q": 19, "nx": 175, "ny": 190, "nz": 201, "dynamics": "bgk",
         "storage": "f64", "steps": 10, "tuned": False},
        # A ragged D3Q27 box with TRT in FP32, default launch shape.
        {"name": "box27_trt_f32", "kind": "box", "q": 27, "nx": 131, "ny": 150, "nz": 97, "dynamics": "trt",
         "storage": "f32", "steps": 20, "tuned": False},
        # The channel past a sphere (D3Q27 TRT, FP16; velocity inlet, pressure outlet, bounce-back
        # side walls, halfway bounce-back sphere), reduced in length; the drag read at the end.
        {"name": "channel_f16", "kind": "channel", "nx": 256, "ny": 96, "nz": 96, "d": 20, "storage": "f16dev",
         "steps": 20, "tuned": True},
        # The porous medium (D3Q27 Smagorinsky-forced BGK, FP16, porosity 0.6), a packing repeated
        # twice along each axis; the FP32 form of a smaller one is drawn.
        {"name": "porous_f16", "kind": "porous", "n": 160, "storage": "f16dev", "steps": 20, "tuned": True},
        # A mix of cavities stepped together by the ensemble engine, then every lattice's fields.
        {"name": "ensemble_mix", "kind": "ensemble", "edges": "32,48,64,96,40,72,48,32,64,56", "storage": "f32",
         "steps": 500},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["cavity2d", "links2", "links3", "monitor", "box", "box", "box16", "box64", "box27", "channel",
                       "porous", "ensemble"])
    if kind == "cavity2d":
        return {"kind": kind, "nx": _log_int(rng, 48, 400), "ny": _log_int(rng, 48, 400),
                "storage": "f64", "steps": rng.randint(50, 100)}
    if kind == "links2":
        return {"kind": "links", "q": 9, "nx": _log_int(rng, 100, 1200), "ny": _log_int(rng, 100, 1200), "nz": 1,
                "storage": rng.choice(["f64", "f32"]), "steps": rng.randint(20, 50)}
    if kind == "links3":
        n = [_log_int(rng, 24, 128) for _ in range(3)]
        return {"kind": "links", "q": rng.choice([19, 27]), "nx": n[0], "ny": n[1], "nz": n[2],
                "storage": rng.choice(["f64", "f32", "f16dev"]), "steps": rng.randint(20, 100)}
    if kind == "monitor":
        n = [_log_int(rng, 32, 128) for _ in range(3)]
        return {"kind": "monitor", "q": 19, "nx": n[0], "ny": n[1], "nz": n[2], "dynamics": "bgk",
                "storage": rng.choice(["f32", "f16dev"]), "steps": rng.randint(5, 20), "tuned": False}
    if kind.startswith("box"):
        n = [_log_int(rng, 40, 256) for _ in range(3)]
        q = 27 if kind == "box27" else 19
        storage = {"box": "f32", "box16": "f16dev", "box64": "f64",
                   "box27": rng.choice(["f32", "f16dev"])}[kind]
        if storage == "f64":
            n = [min(v, 200) for v in n]
        if q == 27:
            n = [min(v, 192) for v in n]
        return {"kind": "box", "q": q, "nx": n[0], "ny": n[1], "nz": n[2],
                "dynamics": rng.choice(["bgk", "trt", "smagorinsky_forced_bgk"]), "storage": storage,
                "steps": rng.randint(5, 20),
                "tuned": rng.random() < 0.5}
    if kind == "channel":
        d = rng.randint(8, 20)
        ny, nz = rng.randint(3 * d, 96), rng.randint(3 * d, 96)
        return {"kind": kind, "nx": rng.randint(96, 256), "ny": ny, "nz": nz, "d": d,
                "storage": "f16dev", "steps": rng.randint(10, 20), "tuned": rng.random() < 0.5}
    if kind == "porous":
        return {"kind": kind, "n": 2 * rng.randint(32, 72), "storage": rng.choice(["f32", "f16dev"]),
                "steps": rng.randint(5, 20), "tuned": rng.random() < 0.5}
    edges = [_log_int(rng, 24, 96) for _ in range(rng.randint(3, 10))]
    return {"kind": "ensemble", "edges": ",".join(str(e) for e in edges), "storage": rng.choice(["f32", "f16dev"]),
            "steps": rng.randint(100, 300)}


# ---- inputs ------------------------------------------------------------------------------------

def _fields(core, seed, device="cuda"):
    """rho [n] and u [3][n] (FP64, on the device) of a Taylor-Green flow with seeded amplitude and
    phases and a little noise."""
    g = torch.Generator(device="cpu").manual_seed(int(seed) % (1 << 62))
    r = torch.rand(8, generator=g, dtype=torch.float64)
    u0 = 0.03 + 0.02 * float(r[0])
    ph = [2 * math.pi * float(r[1 + a]) for a in range(3)]
    nx, ny, nz = core
    x = (2 * math.pi / nx * torch.arange(nx, dtype=torch.float64, device=device) + ph[0])[:, None, None]
    y = (2 * math.pi / ny * torch.arange(ny, dtype=torch.float64, device=device) + ph[1])[None, :, None]
    z = (2 * math.pi / nz * torch.arange(nz, dtype=torch.float64, device=device) + ph[2])[None, None, :]
    u = torch.zeros((3, nx, ny, nz), dtype=torch.float64, device=device)
    rho = torch.ones((nx, ny, nz), dtype=torch.float64, device=device)
    if nz > 1:
        u[0] = u0 * torch.sin(x) * torch.cos(y) * torch.cos(z)
        u[1] = -u0 * torch.cos(x) * torch.sin(y) * torch.cos(z)
        rho += 3 * u0 * u0 / 16 * (torch.cos(2 * x) + torch.cos(2 * y)) * (torch.cos(2 * z) + 2)
    else:
        u[0] = u0 * (torch.sin(x) * torch.cos(y))
        u[1] = -u0 * (torch.cos(x) * torch.sin(y))
        rho += 3 * u0 * u0 / 4 * (torch.cos(2 * x) + torch.cos(2 * y))
    gd = torch.Generator(device=device).manual_seed(int(seed) % (1 << 62))
    u[:2] += 1e-3 * (torch.rand((2, nx, ny, nz), generator=gd, dtype=torch.float64, device=device) - 0.5)
    return rho.reshape(-1), u.reshape(3, -1)


def _omega(seed):
    return 1.1 + 0.6 * float(np.random.default_rng([int(seed) % (1 << 62), 3]).random())


def _cavity_material(core):
    """Fluid (1) inside a layer of walls (2) with the lid (3) at the top of the y axis."""
    mat = np.full(core, 2, np.int32)
    inner = tuple(slice(1, -1) if n > 1 else slice(None) for n in core)
    mat[inner] = 1
    mat[:, -1, :] = 3
    return mat


class _Device:
    """A range of a lattice's device memory for torch.as_tensor, which keeps this object and with it
    the lattice for as long as a view of the memory is held."""

    def __init__(self, lat, ptr, count, typestr):
        self.lat = lat
        self.__cuda_array_interface__ = {"shape": (count,), "typestr": typestr, "data": (ptr, False), "version": 3,
                                         "strides": None}


class _Lattice:
    """A lattice and one flat tensor over all its population columns."""

    def __init__(self, lat):
        info = lat.info()
        self.lat = lat
        ptr, shift = lat.population_ptr(0)
        self.size = _BYTES[lat.storage]
        self.base = ptr - lat.population_shift(0) * self.size if shift == 0 else ptr
        self.flat = torch.as_tensor(_Device(lat, self.base, lat.q * int(info.column_stride), _TYPE[lat.storage]),
                                    device="cuda")
        self.core = lat.core[: lat.d]
        sy = info.padded[2] if lat.d == 3 else 1
        sx = info.padded[1] * sy
        self.strides = (sx, sy, 1)[: lat.d]
        self.first = sum(self.strides)

    def populations(self):
        """The core cells of every population column, as views (no copies)."""
        out = []
        for i in range(self.lat.q):
            ptr, shift = self.lat.population_ptr(i)
            if shift:
                raise RuntimeError("the columns are not mapped twice: no contiguous run to view")
            out.append(self.flat.as_strided(self.core, self.strides, (ptr - self.base) // self.size + self.first))
        return out


def _force(case):
    return (1e-4, 0.0, 0.0) if case.get("dynamics") == "smagorinsky_forced_bgk" else (0.0, 0.0, 0.0)


def _solid(n, seed):
    half = configs.porous_spheres(n // 2, seed=int(seed) % (1 << 31))
    return np.tile(half, (2, 2, 2))


def _lid(seed):
    return 0.04 + 0.04 * float(np.random.default_rng([int(seed) % (1 << 62), 5]).random())


def _requests(case, seed):
    """(edge, omega) of every cavity of the mix: Reynolds numbers log-uniform over [10, 1000]."""
    rng = np.random.default_rng([int(seed) % (1 << 62), 7])
    out = []
    for e in (int(v) for v in case["edges"].split(",")):
        re = math.exp(rng.uniform(math.log(10.0), math.log(1000.0)))
        out.append((e, 1.0 / (3.0 * 0.05 * e / re + 0.5)))
    return out


def prepare(case, seed):
    kind = case["kind"]
    state = {"steps": case["steps"], "kind": kind}
    if kind == "ensemble":
        reqs = [lbx.make_request((e, e, e), w, 0.05, tolerance=0.0, max_steps=1 << 40)
                for e, w in _requests(case, seed)]
        foot = sum(lbx.Ensemble.footprint_of(19, case["storage"], r) for r in reqs)
        ens = lbx.Ensemble(19, case["storage"], slab_bytes=foot + (1 << 20), max_lattices=len(reqs))
        state["ens"] = ens
        state["slots"] = [ens.admit(r) for r in reqs]
        return state
    if kind == "channel":
        extent = (case["nx"], case["ny"], case["nz"])
        lat, _ = configs.channel_sphere(case["storage"], extent, u_peak=_lid(seed), d=case["d"])
    elif kind == "porous":
        lat = configs.porous_medium(_solid(case["n"], seed), case["storage"], force=1e-4)
    elif kind == "cavity2d":
        core = (case["nx"], case["ny"], 1)
        mat = _cavity_material(core)
        lat = lbx.BlockLattice(9, core, (0, 0, 0), case["storage"])
        lat.define_dynamics("bgk", omega=_omega(seed))
        lat.set_cell_dynamics(np.where(mat == 1, lbx.CELL_BULK, lbx.CELL_NONE).astype(np.uint8))
        vals = np.zeros((mat.size, 4))
        vals[mat.reshape(-1) == 3, 0] = _lid(seed)
        lat.set_interpolated_boundary(lbx.FD_VELOCITY, mat.reshape(core[:2]), 2, vals)
        lat.set_interpolated_boundary(lbx.FD_VELOCITY, mat.reshape(core[:2]), 3, vals)
        rho, u = _fields(core, seed)
        rho, u = rho.cpu().numpy(), u[:2].cpu().numpy()
        lat.ini_equilibrium(rho, u)
        lat.post_process()
    else:
        core = (case["nx"], case["ny"], case["nz"])
        q = case["q"]
        d = 2 if q == 9 else 3
        periodic = (0, 0, 0) if kind == "links" else (1, 1, 1 if d == 3 else 0)
        lat = lbx.BlockLattice(q, core, periodic, case["storage"])
        lat.define_dynamics(case.get("dynamics", "bgk"), omega=_omega(seed), smagorinsky=0.12, force=_force(case))
        if kind == "links":
            mat = _cavity_material(core)
            lat.set_cell_dynamics(np.where(mat == 1, lbx.CELL_BULK, lbx.CELL_NONE).astype(np.uint8))
            lat.set_bouzidi_boundary(mat, 1, (2, 3), wall_velocity=[(0, 0, 0), (_lid(seed), 0, 0)])
        rho, u = _fields(core, seed)
        lat.ini_equilibrium(rho.cpu().numpy(), u[:d].cpu().numpy())
        if kind == "links":
            lat.post_process()
    if case.get("tuned"):
        lat.autotune(steps=3)
    state["lat"] = _Lattice(lat)
    state["lattice"] = lat
    return state


def run(state):
    kind, steps = state["kind"], state["steps"]
    if kind == "ensemble":
        ens = state["ens"]
        ens.run(steps)
        fields = [ens.moments(s) for s in state["slots"]]
        return [[torch.from_numpy(v).float() for v in f] for f in fields]  # single-precision lattices
    lat = state["lattice"]
    if kind == "monitor":
        seen = []
        for _ in range(steps):
            lat.collide_and_stream(1, statistics=True)
            s = lat.get_statistics()
            seen.append((s["average_rho"], s["average_energy"], s["max_u"]))
        return {"f": state["lat"].populations(), "seen": np.array(seen, np.float32)}
    lat.collide_and_stream(steps)
    if kind == "links":
        residual = lat.reduce(lbx.REDUCE_RESIDUAL).astype(np.float32)
        return {"f": state["lat"].populations(), "residual": residual}
    if kind == "channel":
        return {"f": state["lat"].populations(), "force": lat.boundary_force(0).astype(np.float32)}
    return {"f": state["lat"].populations()}


# ---- what a pass cannot do without ---------------------------------------------------------------

def _shape(case):
    """(q, cells that are stepped) of a case."""
    kind = case["kind"]
    if kind == "porous":
        return 27, 0.6 * case["n"] ** 3
    if kind == "channel":
        return 27, float(case["nx"] * (case["ny"] - 2) * (case["nz"] - 2) - math.pi * case["d"] ** 3 / 6)
    if kind == "cavity2d":
        return 9, float(case["nx"] * case["ny"])
    if kind == "ensemble":
        return 19, float(sum(int(e) ** 3 for e in case["edges"].split(",")))
    if kind == "links":
        inner = (case["nx"] - 2) * (case["ny"] - 2) * (case["nz"] - 2 if case["q"] != 9 else 1)
        return case["q"], float(inner)
    return case["q"], float(case["nx"] * case["ny"] * case["nz"])


def work(case):
    """Every population read once and written once a pass; one collision per cell and step."""
    q, cells = _shape(case)
    kind = case["kind"]
    dyn = {"porous": "smagorinsky_forced_bgk", "channel": "trt"}.get(kind, case.get("dynamics", "bgk"))
    nbytes = 2.0 * q * _BYTES[case["storage"]] * cells
    if kind == "ensemble":
        nbytes += 32.0 * cells  # rho and u of every cell, read out in FP64
    return {"bytes": nbytes, "flops": _FLOPS[dyn] * q * cells * case["steps"]}


# ---- the same outputs in 64 bits -------------------------------------------------------------------

def _equilibrium(q, rho, u):
    """f_i^eq - w_i of every direction; rho [n...], u [3][n...]."""
    usq = (u * u).sum(0)
    out = []
    for c in _C[q]:
        w = _weight(q, c)
        cu = sum(c[a] * u[a] for a in range(3) if c[a]) if any(c) else torch.zeros_like(rho)
        out.append(w * (rho * (1 + 3 * cu + 4.5 * cu * cu - 1.5 * usq) - 1))
    return torch.stack(out)


def _moments(q, f, force=(0.0, 0.0, 0.0)):
    c = torch.tensor(_C[q], dtype=torch.float64, device=f.device)
    rho = f.sum(0) + 1
    u = torch.tensordot(c.T.contiguous(), f, dims=1) / rho
    for a in range(3):
        if force[a]:
            u[a] += 0.5 * force[a]
    return rho, u


def _collide(q, f, dynamics, omega, force=(0.0, 0.0, 0.0), magic=0.25, smagorinsky=0.12):
    rho, u = _moments(q, f, force)
    feq = _equilibrium(q, rho, u)
    c = _C[q]
    if dynamics == "trt":
        opp = [c.index(tuple(-v for v in k)) for k in c]
        omega2 = 1 / (magic / (1 / omega - 0.5) + 0.5)
        fo, eo = f[opp], feq[opp]
        out = f - omega * 0.5 * ((f + fo) - (feq + eo)) - omega2 * 0.5 * ((f - fo) - (feq - eo))
        return out, rho, u
    w = omega
    if dynamics == "smagorinsky_forced_bgk":
        ud = u.clone()
        for a in range(3):
            ud[a] -= 0.5 * force[a]
        n2 = torch.zeros_like(rho)
        for a in range(3):
            for b in range(a, 3):
                pi = sum(k[a] * k[b] * f[i] for i, k in enumerate(c) if k[a] * k[b])
                pi = pi - rho * ud[a] * ud[b] + 0.5 * rho * (force[a] * ud[b] + ud[a] * force[b])
                if a == b:
                    pi = pi - (rho - 1) / 3
                n2 += pi * pi * (1 if a == b else 2)
        tau = 1 / omega
        pre = smagorinsky ** 2 * 18 * math.sqrt(2.0)
        w = 1 / (tau + 0.5 * (torch.sqrt(tau * tau + pre / rho * torch.sqrt(n2)) - tau))
    out = f + w * (feq - f)
    if any(force):
        for i, k in enumerate(c):
            cu = sum(k[a] * u[a] for a in range(3))
            s = sum(((k[a] - u[a]) * 3 + 9 * cu * k[a]) * force[a] for a in range(3))
            out[i] += rho * (1 - 0.5 * w) * _weight(q, k) * s
    return out, rho, u


class _Exact:
    """The lattice in 64 bits: population i of padded cell n in f[i, n], every column cyclic over the
    padded cells rounded up to 2 MiB of the storage type, so that what streams out of the core, into
    walls and padding and back is where the library's columns have it."""

    def __init__(self, q, core, periodic, size, solid=None, wall=None, device="cuda"):
        self.q, self.core, self.device = q, core, device
        d = 2 if q == 9 else 3
        self.pad = (core[0] + 2, core[1] + 2, core[2] + 2 if d == 3 else 1)
        self.strides = (self.pad[1] * self.pad[2], self.pad[2], 1)
        n = self.pad[0] * self.strides[0]
        gran = (2 << 20) // size
        self.f = torch.zeros((q, -(-n // gran) * gran), dtype=torch.float64, device=device)
        c = _C[q]
        self.off = [sum(k[a] * self.strides[a] for a in range(3)) for k in c]
        ax = [torch.arange(v, device=device) for v in core]
        pz = 1 if d == 3 else 0
        x, y, z = torch.meshgrid(*ax, indexing="ij")
        flat = ((x + 1) * self.strides[0] + (y + 1) * self.strides[1] + z + pz).reshape(-1)
        pos = torch.stack([x.reshape(-1), y.reshape(-1), z.reshape(-1)])
        fluid = torch.ones_like(flat, dtype=torch.bool) if solid is None else ~solid.reshape(-1)
        self.all, self.cells = flat, flat[fluid]
        ext = torch.tensor(core, device=device)[:, None]
        per = torch.tensor([bool(v) for v in periodic], device=device)[:, None]
        self.ghost, self.link = [], []
        solid_flat = None if solid is None else solid.reshape(-1)
        for i, k in enumerate(c):
            kk = torch.tensor(k, device=device)[:, None]
            t = pos + kk
            out = (t < 0) | (t >= ext)
            wrapped = torch.where(out & per, (t + ext) % ext, t)
            inside = ~(out & ~per).any(0)
            # what crosses a periodic face: the padding slot one step before the cell it reaches
            sel = fluid & inside & out.any(0)
            src = wrapped[:, sel] - kk
            slot = (src[0] + 1) * self.strides[0] + (src[1] + 1) * self.strides[1] + src[2] + pz
            self.ghost.append((flat[sel], slot))
            if solid_flat is None or i == 0:
                self.link.append(None)
                continue
            w = wrapped.clamp(min=0)
            at = (torch.minimum(w[0], ext[0] - 1) * core[1] + torch.minimum(w[1], ext[1] - 1)) * core[2] \
                + torch.minimum(w[2], ext[2] - 1)
            hit = fluid & inside & solid_flat[at]
            term = 6 * _weight(q, k) * k[0] * wall.reshape(-1)[at[hit]] if wall is not None else 0.0
            self.link.append((flat[hit], term))

    def post_process(self):
        c = _C[self.q]
        old = self.f.clone()
        for i, k in enumerate(c):
            if self.link[i] is not None:
                at, term = self.link[i]
                self.f[c.index(tuple(-v for v in k)), at] = old[i, at + self.off[i]] - term

    def step(self, dynamics, omega, force=(0.0, 0.0, 0.0)):
        c = _C[self.q]
        f, rho, u = _collide(self.q, self.f[:, self.cells], dynamics, omega, force)
        self.f[:, self.cells] = f
        moved = torch.empty_like(self.f)
        sent = []
        for i in range(self.q):
            src, slot = self.ghost[i]
            self.f[i, slot] = self.f[i, src]
            if self.link[i] is not None:
                at, term = self.link[i]
                sent.append((c.index(tuple(-v for v in c[i])), at + self.off[i], self.f[i, at] - term))
        for i, slot, v in sent:
            self.f[i, slot] = v
        for i in range(self.q):
            moved[i] = torch.roll(self.f[i], self.off[i])
        self.f = moved
        return rho, u

    def populations(self):
        core = self.core[: 2 if self.q == 9 else 3]
        return [self.f[i, self.all].reshape(core) for i in range(self.q)]


def _exact_cavity(edge, omega, steps, device):
    """rho and u of a box cavity at rest whose lid (+y) moves along x: walls half a cell outside."""
    core = (edge + 2,) * 3
    mat = torch.from_numpy(_cavity_material(core)).to(device)
    lid = torch.zeros(core, dtype=torch.float64, device=device)
    lid[1:-1, -1, 1:-1] = 0.05
    # a link through the lid and a side wall at once leaves through the lid
    for at in (0, -1):
        lid[at, -1, :] = 0.05
        lid[:, -1, at] = 0.05
    lat = _Exact(19, core, (0, 0, 0), 4, mat != 1, lid, device)
    lat.post_process()
    for _ in range(steps):
        lat.step("bgk", omega)
    rho, u = _moments(19, lat.f[:, lat.cells])
    return [rho, u]


def exact(case, seed):
    kind, storage = case["kind"], case["storage"]
    if kind in ("channel", "cavity2d"):
        return None  # the boundary schemes' restatement is the test oracle's business
    device = "cuda" if torch.cuda.is_available() else "cpu"
    if kind == "ensemble":
        return [_exact_cavity(e, w, case["steps"], device) for e, w in _requests(case, seed)]
    if kind == "porous":
        solid = torch.from_numpy(_solid(case["n"], seed)).to(device)
        lat = _Exact(27, (case["n"],) * 3, (1, 1, 1), _BYTES[storage], solid, None, device)
        for _ in range(case["steps"]):
            lat.step("smagorinsky_forced_bgk", 1 / (3 * 0.05 + 0.5), (1e-4, 0.0, 0.0))
        return {"f": lat.populations()}
    q, core = case["q"], (case["nx"], case["ny"], case["nz"])
    rho, u = _fields(core, seed, device)
    if kind == "links":
        mat = torch.from_numpy(_cavity_material(core)).to(device)
        wall = (mat == 3).double() * _lid(seed)
        lat = _Exact(q, core, (0, 0, 0), _BYTES[storage], mat != 1, wall, device)
    else:
        lat = _Exact(q, core, (1, 1, 1 if q != 9 else 0), _BYTES[storage], None, None, device)
    lat.f[:, lat.all] = _equilibrium(q, rho, u)
    lat.post_process()
    seen = []
    for _ in range(case["steps"]):
        rho, u = lat.step(case.get("dynamics", "bgk"), _omega(seed), _force(case))
        if kind == "monitor":
            usq = (u * u).sum(0)
            seen.append((float(rho.mean()), float(0.5 * usq.mean()), float(usq.max().sqrt())))
    out = {"f": lat.populations()}
    if kind == "monitor":
        out["seen"] = np.array(seen)
    if kind == "links":
        _, u = _moments(q, lat.f[:, lat.cells])
        u2 = (u * u).sum(0)
        out["residual"] = np.array([float(u2.sum().sqrt()), float(u2.sum().sqrt()), float(u2.max().sqrt())])
    return out
