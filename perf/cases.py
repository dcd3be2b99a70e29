"""What a user of this package has it do, as cases that can be timed.

A case is a dict of plain values.  Its "op" says which public entry point it
goes through:

  steps    Lattice.step: a solve advanced between two outputs (the cavity,
           Taylor-Green, channel and sphere configurations), with the drag of
           the sphere at the end where there is one
  energy   Lattice.step_moments: the same, with the kinetic energy and the
           mass recorded on the way
  sweep    DeviceLattice.sweep: a caller's own arrays in the reference's
           layout (row pitch l + 2), one call per time step, as a driver
           that keeps its own time loop makes it
  batch    Batch.step: a parameter sweep of small and middle lattices
  serve    Server.run: a burst of solve requests, from admission to results
  diag     Lattice.moments, dissipation, profile and slice of one state

listed() holds the configurations the package is built around and the ragged
sizes and options beside them; draw() gives more of the same ranges.
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

from bgk3d_gpu_b200 import cases as CS
from bgk3d_gpu_b200 import serve as SV
from bgk3d_gpu_b200.lattice import Batch, DeviceLattice, Lattice

DTYPE = {"f64": torch.float64, "f32": torch.float32, "f16": torch.float16, "bf16": torch.bfloat16,
         "f32_f64": torch.float32}
BYTES = {"f64": 8, "f32": 4, "f16": 2, "bf16": 2, "f32_f64": 4}
SCALE = {"f16": 256.0}          # the storage scale make_lattice gives FP16 lattices
BATCH_SIDES = (32, 48, 64, 96, 128, 160)
SERVE_SIDES = (32, 40, 54, 72, 96, 128)
OPS_PER_UPDATE = 250            # additions and multiplications of one collision

# velocities, weights and opposite populations of the D3Q19 set (01..19)
CX = (1, 1, 1, 1, 1, 0, 0, 0, 0, -1, -1, -1, -1, -1, 0, 0, 0, 0, 0)
CY = (-1, 0, 1, 0, 0, 0, 1, 1, 1, -1, 0, 1, 0, 0, 0, -1, -1, -1, 0)
CZ = (0, -1, 0, 1, 0, 1, 1, 0, -1, 0, -1, 0, 1, 0, -1, -1, 0, 1, 0)
OPP = (11, 12, 9, 10, 13, 14, 15, 16, 17, 2, 3, 0, 1, 4, 5, 6, 7, 8, 18)
W = tuple((1 / 3, 1 / 18, 1 / 36)[abs(x) + abs(y) + abs(z)] for x, y, z in zip(CX, CY, CZ))


def _case(name, op, kind, bcase, l, m, n, steps, pattern="ab", fast=False, every=0, count=0):
    return dict(name=name, op=op, kind=kind, bcase=bcase, l=l, m=m, n=n, steps=steps, pattern=pattern,
                fast=fast, every=every, count=count)


def listed():
    return [
        # the lid-driven cavity configuration: double precision, 128^3
        _case("cavity_f64_128", "steps", "f64", "driven", 128, 128, 128, 100),
        # the Taylor-Green configuration (the headline benchmark): 256^3, energy sampled along the decay
        _case("tgv_f32_256", "energy", "f32", "periodic", 256, 256, 256, 100, every=50),
        # the same in shifted half precision with the fused collision
        _case("tgv_f16_256_fast", "steps", "f16", "periodic", 256, 256, 256, 100, fast=True),
        # the sphere configuration: inflow, outflow, an obstacle, drag sampled every so many steps
        _case("sphere_f32_512", "steps", "f32", "inflow", 512, 256, 256, 60),
        # a sphere in the in-place pattern and bfloat16: the smallest footprint
        _case("sphere_bf16_aa_256", "steps", "bf16", "inflow", 256, 128, 128, 100, pattern="aa"),
        # a force-driven channel of odd sides: ragged rows in every direction
        _case("channel_f32_199", "steps", "f32", "channel", 199, 83, 61, 100),
        # in place, single precision: a lattice chosen for its footprint
        _case("cavity_f32_aa_192", "steps", "f32", "driven", 192, 192, 192, 60, pattern="aa"),
        # a small periodic solve, where launches count
        _case("small_f32_32", "steps", "f32", "periodic", 32, 32, 32, 500),
        # energy and mass of every step, as a monitored run records them
        _case("monitored_f32_160", "energy", "f32", "periodic", 160, 160, 160, 64, every=1),
        # a driver with its own arrays and time loop
        _case("sweep_f32_256", "sweep", "f32", "driven", 256, 256, 256, 20),
        # the batched parameter sweep: half Kida vortices, half forced channels, sides 32 to 160
        _case("batch_f32_24", "batch", "f32", "mixed", 160, 160, 160, 48, count=24),
        # a burst of solve requests of every kind of case
        _case("serve_8", "serve", "mixed", "mixed", 128, 128, 128, 600, count=8),
    ]


def draw(rng):
    op = rng.choice(["steps"] * 6 + ["energy", "sweep", "batch", "serve", "diag"])
    kind = rng.choice(["f32", "f32", "f32", "f64", "f16", "bf16"])
    fast = kind != "f64" and rng.random() < 0.4
    if op == "batch":
        return _plain(_case("", op, kind if kind in ("f64", "f32") else "f32", "mixed", rng.choice(BATCH_SIDES[2:]), 0, 0,
                            rng.choice((20, 32, 48)), fast=fast and kind == "f32", count=rng.randint(6, 24)))
    if op == "serve":
        return _plain(_case("", op, "mixed", "mixed", rng.choice(SERVE_SIDES[2:]), 0, 0, rng.randint(500, 700),
                            count=rng.randint(4, 8), fast=fast))
    side = math.exp(rng.uniform(math.log(32), math.log(256)))
    l, m, n = (max(24, min(320, int(round(side * math.exp(rng.uniform(-0.35, 0.35)))))) for _ in range(3))
    if rng.random() < 0.4:
        l = l // 32 * 32 if l >= 32 else 32
    bcase = rng.choice(["driven", "periodic", "channel", "inflow"])
    if op == "diag":
        kind, bcase, fast = rng.choice(["f32", "f64"]), rng.choice(["periodic", "channel", "driven"]), False
        return _plain(_case("", op, kind, bcase, l, m, n, 0))
    if op == "sweep" and bcase == "inflow":
        bcase = "periodic"
    pattern = "aa" if op == "steps" and rng.random() < 0.3 else "ab"
    most = int(1.2e9 / (l * m * n) * 4 / BYTES[kind])
    steps = max(8, min(500, int(most * math.exp(rng.uniform(-1.5, 0)))))
    if op == "sweep":
        steps = min(steps, 40)
    if pattern == "aa" or bcase == "inflow" or op == "sweep":
        steps += steps % 2      # a state that can be read, solid nodes and arrays where they were
    every = rng.choice([1, 1, 5, 10]) if op == "energy" else 0
    if every:
        steps = max(every, steps // every * every)
        steps += every * (bcase == "inflow" and steps % 2)
    return _plain(_case("", op, kind, bcase, l, m, n, steps, pattern=pattern, fast=fast, every=every))


def _plain(case):
    del case["name"]
    return case


# --------------------------------------------------------------------- inputs
def _rng(seed):
    return np.random.default_rng([int(seed), 1907])


def _physics(case, rng):
    """Lattice keyword arguments of the case's flow; viscosities and speeds as the configurations have them."""
    kw = dict(omega=1.0 / rng.uniform(0.55, 0.8))
    if case["bcase"] == "driven":
        kw["lid_force"] = rng.uniform(0.05, 0.1) / 6.0
    elif case["bcase"] == "channel":
        kw.update(force_mode=1, force=(rng.uniform(0.5, 2.0) * 1e-7, 0.0, 0.0))
    elif case["bcase"] == "inflow":
        kw["u_inflow"] = rng.uniform(0.03, 0.05)
    return kw


def _sphere(case):
    """(centre, radius^2) of the obstacle of an inflow case, or None where the lattice is too thin for one."""
    if case["bcase"] != "inflow" or min(case["l"], case["m"], case["n"]) < 24:
        return None
    d = min(case["l"], case["m"], case["n"]) / 6.0
    return (float(case["l"] // 4 + 2), float(case["m"] // 2), float(case["n"] // 2)), (d / 2.0) ** 2


def _drag_box(case):
    return CS.drag_box(CS.sphere_bbox(case["l"], case["m"], case["n"], 2.0 * math.sqrt(_sphere(case)[1]), _sphere(case)[0]))


def _flow(l, m, n, rng, dev, u0=0.04):
    """A smooth flow of a few Fourier modes, density about 1: fields (n, m, l) in FP64."""
    axes = [torch.arange(s, dtype=torch.float64, device=dev) * (2.0 * math.pi / s) for s in (n, m, l)]
    z, y, x = axes[0][:, None, None], axes[1][None, :, None], axes[2][None, None, :]
    out = []
    for amp in (0.01, u0, u0, u0):
        f = torch.zeros((n, m, l), dtype=torch.float64, device=dev)
        for _ in range(2):
            kx, ky, kz = (int(v) for v in rng.integers(1, 4, 3))
            px, py, pz = rng.uniform(0, 2 * math.pi, 3)
            f += (0.5 * amp * rng.uniform(0.5, 1.0)) * (torch.sin(kx * x + px) * torch.cos(ky * y + py)) * torch.cos(kz * z + pz)
        out.append(f)
    out[0] += 1.0
    return out


def _equilibrium(rho, ux, uy, uz, d):
    """f_d^eq - w_d (shifted storage) in FP64."""
    cu = CX[d] * ux + CY[d] * uy + CZ[d] * uz
    q = 3.0 * cu + 4.5 * cu * cu - 1.5 * (ux * ux + uy * uy + uz * uz)
    return W[d] * (rho - 1.0) + W[d] * rho * q


class _Memory:
    """Device memory of an object that owns it (kept alive as long as a tensor views it)."""

    def __init__(self, owner, ptr, shape, strides, typestr):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": shape, "typestr": typestr, "data": (ptr, False), "version": 3,
                                         "strides": strides}


class _Views:
    """The interior of a library-owned lattice's current populations as tensors, through bgk_lattice_arrays."""

    def __init__(self, lat):
        self.lat, self.seen = lat, {}
        self.ptrs = (ctypes.c_void_p * 19)()
        nx, ny = ctypes.c_longlong(), ctypes.c_longlong()
        lat.L.bgk_lattice_arrays(lat.h, self.ptrs, ctypes.byref(nx), ctypes.byref(ny))
        kind = {0: "f64", 1: "f32", 2: "f16", 3: "bf16", 4: "f32"}[lat.kind]
        self.dtype, self.es = DTYPE[kind], BYTES[kind]
        self.typestr = {8: "<f8", 4: "<f4", 2: "<i2"}[self.es]
        self.strides = (nx.value * ny.value * self.es, nx.value * self.es, self.es)

    def _view(self, ptr):
        v = self.seen.get(ptr)
        if v is None:
            at = ptr + sum(self.strides)          # node (1, 1, 1)
            mem = _Memory(self.lat, at, (self.lat.n, self.lat.m, self.lat.l), self.strides, self.typestr)
            v = torch.as_tensor(mem, device="cuda")
            v = self.seen[ptr] = v.view(self.dtype) if v.dtype != self.dtype else v
        return v

    def __call__(self):
        self.lat.L.bgk_lattice_arrays(self.lat.h, self.ptrs, None, None)
        return [self._view(p) for p in self.ptrs]

    def whole(self):
        """All populations as one (19, n, m, l) tensor; the arrays are evenly spaced after an even step count."""
        self.lat.L.bgk_lattice_arrays(self.lat.h, self.ptrs, None, None)
        key = (self.ptrs[0], "all")
        if key not in self.seen:
            step = self.ptrs[1] - self.ptrs[0]
            if any(self.ptrs[d] - self.ptrs[0] != d * step for d in range(19)):
                raise RuntimeError("populations are not evenly spaced")
            mem = _Memory(self.lat, self.ptrs[0] + sum(self.strides), (19, self.lat.n, self.lat.m, self.lat.l),
                          (step,) + self.strides, self.typestr)
            v = torch.as_tensor(mem, device="cuda")
            self.seen[key] = v.view(self.dtype) if v.dtype != self.dtype else v
        return self.seen[key]


def _new_lattice(case, seed):
    """A lattice of the case with a seeded smooth flow in it, and its views."""
    rng = _rng(seed)
    kw = _physics(case, rng)
    scale = SCALE.get(case["kind"], 1.0)
    lat = Lattice(case["l"], case["m"], case["n"], kind=case["kind"], bcase=case["bcase"], pattern=case["pattern"],
                  fast=case["fast"], scale=scale, **kw)
    sph = _sphere(case)
    if sph:
        lat.set_sphere(*sph)
    views = _Views(lat)
    flow = _flow(case["l"], case["m"], case["n"], rng, "cuda")
    if case["pattern"] == "aa" and case["bcase"] == "inflow":
        # the in-place pattern prepares its outflow plane when a state is loaded
        full = torch.zeros((19, case["n"] + 2, case["m"] + 2, case["l"] + 2), dtype=DTYPE[case["kind"]], device="cuda")
        for d in range(19):
            e = _equilibrium(*flow, d)
            full[d, 1:-1, 1:-1, 1:-1] = e if full.element_size() > 2 else e.float() * scale
        host = full.cpu()
        lat.upload(host.view(torch.int16).numpy().view(np.uint16) if full.element_size() == 2 else host.numpy())
    else:
        lat.init_flow("rest")
        for d, v in enumerate(views()):
            e = _equilibrium(*flow, d)
            v.copy_(e if v.element_size() > 2 else e.float() * scale)
    return lat, views


def _batch_cases(case):
    """The lattices of a batch: sides up to the case's, alternating Kida-like periodic and forced channel."""
    sides = [s for s in BATCH_SIDES if s <= case["l"]]
    out = []
    for i in range(case["count"]):
        s = sides[(i // 2) % len(sides)]
        out.append(_case("", "steps", case["kind"], "periodic" if i % 2 == 0 else "channel", s, s, s, case["steps"],
                         fast=case["fast"]))
    return out


def _requests(case, seed):
    rng = _rng(seed)
    sides = [s for s in SERVE_SIDES if s <= case["l"]]
    out = []
    for i in range(case["count"]):
        out.append(SV.Request(i, 0.0, ("ldc", "tgv", "sphere")[i % 3], sides[(5 * i + 1) % len(sides)], case["steps"] + 4 * i,
                              float(rng.uniform(0.55, 0.8)), "f32" if i % 2 == 0 else "f16", case["fast"]))
    return out


def prepare(case, seed):
    op = case["op"]
    if op == "serve":
        return {"case": case, "server": SV.Server(), "trace": _requests(case, seed)}
    if op == "batch":
        made = [_new_lattice(c, seed * 1000 + i) for i, c in enumerate(_batch_cases(case))]
        return {"case": case, "batch": Batch([lat for lat, _ in made]), "views": [v for _, v in made]}
    if op == "sweep":
        rng = _rng(seed)
        kw = _physics(case, rng)
        scale = SCALE.get(case["kind"], 1.0)
        lat = DeviceLattice(case["l"], case["m"], case["n"], kind=case["kind"], bcase=case["bcase"], fast=case["fast"],
                            scale=scale, **kw)
        flow = _flow(case["l"], case["m"], case["n"], rng, "cuda")
        for d in range(19):
            e = _equilibrium(*flow, d)
            lat.A[d, 1:-1, 1:-1, 1:-1].copy_(e if lat.A.element_size() > 2 else e.float() * scale)
        return {"case": case, "lat": lat}
    lat, views = _new_lattice(case, seed)
    state = {"case": case, "lat": lat, "views": views}
    if op == "steps":
        state["box"] = _drag_box(case) if _sphere(case) else None
    return state


# ------------------------------------------------------------------- one pass
def run(state):
    case = state["case"]
    op = case["op"]
    if op == "steps":
        lat = state["lat"]
        lat.step(case["steps"])
        out = {"populations": state["views"]()}
        if state["box"]:
            out["draglift"] = lat.draglift(state["box"])
        return out
    if op == "energy":
        moments = state["lat"].step_moments(case["steps"], every=case["every"])
        return {"populations": state["views"](), "moments": moments}
    if op == "sweep":
        state["lat"].step(case["steps"])
        return {"populations": state["lat"].A[:, 1:-1, 1:-1, 1:-1]}
    if op == "batch":
        state["batch"].step(case["steps"])
        return {"populations": [v.whole() for v in state["views"]]}
    if op == "serve":
        done, _ = state["server"].run(state["trace"])
        done.sort(key=lambda r: r["rid"])
        return {"moments": np.array([r["moments"] for r in done]),
                "draglift": np.array([r["draglift"] for r in done if "draglift" in r])}
    lat = state["lat"]
    return {"moments": lat.moments(), "dissipation": lat.dissipation(0.01),
            "profile": lat.profile(2, case["l"] // 2 + 1, case["m"] // 2 + 1), "slice": lat.slice(0, case["n"] // 2 + 1)}


def work(case):
    op = case["op"]
    if op == "batch":
        each = [c["l"] ** 3 for c in _batch_cases(case)]
        return {"bytes": 2 * 19 * BYTES[case["kind"]] * sum(each), "flops": OPS_PER_UPDATE * case["steps"] * sum(each)}
    if op == "serve":
        nodes = [(r.side ** 3 * (2 if r.case == "sphere" else 1), BYTES[r.kind], r.steps) for r in _requests(case, 0)]
        return {"bytes": sum(2 * 19 * b * v for v, b, _ in nodes), "flops": sum(OPS_PER_UPDATE * s * v for v, _, s in nodes)}
    nodes = case["l"] * case["m"] * case["n"]
    if op == "diag":
        return {"bytes": 19 * BYTES[case["kind"]] * nodes, "flops": 2 * OPS_PER_UPDATE * nodes}
    return {"bytes": 2 * 19 * BYTES[case["kind"]] * nodes, "flops": OPS_PER_UPDATE * case["steps"] * nodes}


# ------------------------------------------------------------- in 64 bits
class _Exact:
    """The same time steps in FP64 with torch: pull, boundary links, BGK collision."""

    def __init__(self, f, bcase, phys, solid=None):
        self.f, self.bcase, self.phys, self.solid = f, bcase, phys, solid     # f: (19, n, m, l), shifted
        t = lambda v: torch.tensor(v, dtype=torch.float64, device=f.device)   # noqa: E731
        self.c, self.w = t([CX, CY, CZ]), t(W)[:, None, None, None]

    def pulled(self):
        f, bc = self.f, self.bcase
        wall = {"driven": (True, True, True), "channel": (False, False, True)}.get(bc, (False,) * 3)
        out = torch.empty_like(f)
        if bc == "inflow":
            mx, my, mz = torch.tensordot(self.c, f[:, :, :, -1], dims=1)
            sq = mx * mx + my * my + mz * mz
        for d in range(18):
            x, own = out[d], f[OPP[d]]
            x.copy_(torch.roll(f[d], (CZ[d], CY[d], CX[d]), (0, 1, 2)))
            for axis, c in ((2, CX[d]), (1, CY[d]), (0, CZ[d])):
                if wall[2 - axis] and c:
                    face = [slice(None)] * 3
                    face[axis] = 0 if c == 1 else -1
                    x[tuple(face)] = own[tuple(face)]
            if bc == "driven" and CZ[d] == -1 and CX[d]:
                x[-1] += CX[d] * self.phys["lid_force"]
            if bc == "inflow" and CX[d] == 1:
                u = self.phys["u_inflow"]
                x[:, :, 0] = W[d] * (3.0 * u + 3.0 * u * u)
            if bc == "inflow" and CX[d] == -1:
                cu = -mx + CY[d] * my + CZ[d] * mz
                e = W[d] * (3.0 * cu + 4.5 * cu * cu - 1.5 * sq)
                x[:, :, -1] = torch.roll(e, (CZ[d], CY[d]), (0, 1))
            if self.solid is not None:
                x.copy_(torch.where(torch.roll(self.solid, (CZ[d], CY[d], CX[d]), (0, 1, 2)), own, x))
        out[18] = f[18]
        return out

    def velocity(self, f):
        rho = f.sum(0) + 1.0
        return rho, *(torch.tensordot(self.c, f, dims=1) / rho)

    def equilibrium(self, rho, ux, uy, uz):
        cu = torch.tensordot(self.c.T, torch.stack((ux, uy, uz)), dims=1)
        q = 3.0 * cu + 4.5 * cu * cu - 1.5 * (ux * ux + uy * uy + uz * uz)
        return self.w * ((rho - 1.0) + rho * q)

    def step(self, nsteps):
        om, force = self.phys["omega"], self.phys.get("force")
        for _ in range(nsteps):
            x = self.pulled()
            mac = self.velocity(x)
            x -= om * (x - self.equilibrium(*mac))
            if force:
                x += (self.c[0] * force[0])[:, None, None, None] * mac[0]
            if self.solid is not None:
                x = torch.where(self.solid, self.f, x)
            self.f = x

    def _sum(self, v):
        return float((torch.where(self.solid, 0.0, v) if self.solid is not None else v).sum())

    def moments(self):
        rho, u, v, w = self.velocity(self.f)
        return [self._sum(q) for q in (rho, u, v, w, 0.5 * (u * u + v * v + w * w))]

    def draglift(self, box):
        """Momentum exchange with the solid, over the fluid nodes of the box."""
        i0, i1, j0, j1, k0, k1 = box
        n, m, l = self.f[0].shape
        at = (slice(max(k0, 1) - 1, min(k1, n)), slice(max(j0, 1) - 1, min(j1, m)), slice(max(i0, 1) - 1, min(i1, l)))
        out = [0.0, 0.0, 0.0]
        for d in range(18):
            hit = torch.roll(self.solid, (-CZ[d], -CY[d], -CX[d]), (0, 1, 2)) & ~self.solid
            s = float(torch.where(hit, self.f[d], 0.0)[at].sum())
            for a, c in enumerate((CX[d], CY[d], CZ[d])):
                out[a] += 2.0 * c * s
        return out

    def dissipation(self, nu):
        x = self.pulled()
        rho, u, v, w = self.velocity(x)
        neq = x - self.equilibrium(rho, u, v, w)
        p2 = sum((1.0 if a is b else 2.0) * sum(a[d] * b[d] * neq[d] for d in range(18) if a[d] * b[d]) ** 2
                 for a, b in ((CX, CX), (CY, CY), (CZ, CZ), (CX, CY), (CX, CZ), (CY, CZ)))
        out = [self._sum(q) for q in (0.5 * (u * u + v * v + w * w), 2.0 * nu * p2, u * u, v * v, w * w)]
        _, u, v, w = self.velocity(self.f)
        dif = lambda q, ax: 0.5 * (torch.roll(q, -1, ax) - torch.roll(q, 1, ax))  # noqa: E731
        ox, oy, oz = dif(v, 0) - dif(w, 1), dif(w, 2) - dif(u, 0), dif(u, 1) - dif(v, 2)
        ens = 0.5 * (ox * ox + oy * oy + oz * oz)
        inner = [slice(None) if per else slice(1, -1) for per in {
            "periodic": (True, True, True), "channel": (False, True, True), "driven": (False, False, False)}[self.bcase]]
        ens = ens[tuple(inner)]
        return out + [float(ens.sum()), float(ens.numel())]


def _exact_of(case, seed, device):
    """The _Exact of a library-owned lattice's inputs, as _new_lattice makes them."""
    rng = _rng(seed)
    phys = _physics(case, rng)
    flow = _flow(case["l"], case["m"], case["n"], rng, device)
    dt, scale = DTYPE[case["kind"]], SCALE.get(case["kind"], 1.0)
    f = []
    for d in range(19):
        e = _equilibrium(*flow, d)
        f.append((e.float() * scale).to(dt).double() / scale if dt in (torch.float16, torch.bfloat16) else e.to(dt).double())
    f = torch.stack(f)
    sph = _sphere(case)
    return _Exact(f, case["bcase"], phys, _ball(case["l"], case["m"], case["n"], sph, device) if sph else None)


def _ball(l, m, n, sph, device):
    (cx, cy, cz), r2 = sph
    ax = [torch.arange(1, s + 1, dtype=torch.float64, device=device) for s in (n, m, l)]
    return ((ax[2][None, None, :] - cx) ** 2 + (ax[1][None, :, None] - cy) ** 2 + (ax[0][:, None, None] - cz) ** 2) <= r2


def exact(case, seed):
    device = "cuda" if torch.cuda.is_available() else "cpu"
    op = case["op"]
    if device == "cpu" and work(case)["flops"] > 5e9:
        return None
    if op == "serve":
        return _exact_serve(case, seed, device)
    if op == "batch":
        out = []
        for i, c in enumerate(_batch_cases(case)):
            e = _exact_of(c, seed * 1000 + i, device)
            e.step(case["steps"])
            out.append(e.f.cpu())
        return {"populations": out}
    e = _exact_of(case, seed, device)
    if op == "diag":
        rho, u, v, w = e.velocity(e.f)
        i, j, k = case["l"] // 2, case["m"] // 2, case["n"] // 2
        line = torch.stack([torch.arange(case["n"], dtype=torch.float64, device=device) + 0.5]
                           + [q[:, j, i] for q in (u, v, w, rho)], dim=1)
        return {"moments": np.array(e.moments()), "dissipation": np.array(e.dissipation(0.01)), "profile": line,
                "slice": torch.stack([u[k], v[k], w[k]], dim=-1)}
    out = {}
    if op == "energy":
        rows = []
        for _ in range(case["steps"] // case["every"]):
            e.step(case["every"])
            rows.append(e.moments())
        out["moments"] = np.array(rows)
    else:
        e.step(case["steps"])
    if op == "steps" and _sphere(case):
        out["draglift"] = np.array(e.draglift(_drag_box(case)))
    f = e.f * SCALE.get(case["kind"], 1.0)        # storage units, what the arrays hold
    out["populations"] = f if op == "sweep" else list(f)
    return out


def _exact_serve(case, seed, device):
    moments, forces = [], []
    for r in _requests(case, seed):
        c = SV.case_of(r)
        l, m, n = c["l"], c["m"], c["n"]
        ax = [torch.arange(s, dtype=torch.float64, device=device) * (2.0 * math.pi / s) for s in (n, m, l)]
        z, y, x = ax[0][:, None, None], ax[1][None, :, None], ax[2][None, None, :]
        zero = torch.zeros((n, m, l), dtype=torch.float64, device=device)
        flow = [zero + 1.0, zero, zero, zero]
        if r.case == "tgv":
            u0 = c["flow"][1][0]
            flow = [1.0 + 3.0 * (u0 * u0 / 16.0) * (torch.cos(2 * x) + torch.cos(2 * y)) * (torch.cos(2 * z) + 2.0),
                    u0 * torch.sin(x) * torch.cos(y) * torch.cos(z), -u0 * torch.cos(x) * torch.sin(y) * torch.cos(z), zero]
        phys = {"omega": c["omega"], "lid_force": c.get("lid_force", 0.0), "u_inflow": c.get("u_inflow", 0.0)}
        solid = _ball(l, m, n, c["sphere"], device) if r.case == "sphere" else None
        e = _Exact(torch.stack([_equilibrium(*flow, d) for d in range(19)]), c["bcase"], phys, solid)
        e.step(r.steps)
        moments.append(e.moments())
        if solid is not None:
            forces.append(e.draglift(c["drag_box"]))
    return {"moments": np.array(moments), "draglift": np.array(forces)}
