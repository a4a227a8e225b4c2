"""The work a user of this framework has it do, as cases that can be timed and checked.

Each case goes through the public Python binding (``sphmp``), which is a thin layer over the C ABI. A simulation
case is a whole job: the particle records of a scene go up from pinned host memory, are sorted, the boundary
volumes are computed, a few steps run, and every record comes back, as a host program drives the library. A job
starts from the same records in every pass, so that every pass does the same work. The corrector's cases are its
training loop and its inference on device arrays.

``exact`` restates the job in 64 bits with plain torch. Between steps it rounds the state to the 32 bits that the
library's arrays hold, so that the sort of each step sees the same positions.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "sph-multiphase_gb300"))

import sphmp  # noqa: E402
from sphmp import abi, learned, scenes  # noqa: E402

SCHEDULES = {"fused": abi.SCHEDULE_FUSED, "reference": abi.SCHEDULE_REFERENCE, "projectu": abi.SCHEDULE_PROJECTU}
LAYERS = ((48, 128), (128, 128), (128, 128), (128, 4))  # the corrector network
LR = 1e-3


def listed():
    return [
        # an interactive scene: a 4,096-particle dam break with a gas bubble, where launches and latency count
        {"name": "dam_16_fused", "kind": "job", "scene": "dam", "nx": 16, "ny": 16, "nz": 16, "schedule": "fused", "steps": 8},
        # the 32,768-particle two-phase dam break of the benchmark
        {"name": "dam_32_fused", "kind": "job", "scene": "dam", "nx": 32, "ny": 32, "nz": 32, "schedule": "fused", "steps": 8},
        # the 1,048,576-particle three-phase lattice of the benchmark, soft EOS, gas blobs included
        {"name": "blobs_1m_fused", "kind": "job", "scene": "blobs", "nx": 128, "ny": 64, "nz": 128, "schedule": "fused", "steps": 8},
        # three liquids under the reference's EOS in the reference's call order; odd sizes, an odd number of steps
        {"name": "liquids_odd_reference", "kind": "job", "scene": "liquids", "nx": 75, "ny": 41, "nz": 67, "schedule": "reference", "steps": 5},
        # the legacy multiphase step with the drift-tensor force and the XSPH correction
        {"name": "liquids_projectu", "kind": "job", "scene": "liquids", "nx": 96, "ny": 48, "nz": 64, "schedule": "projectu", "steps": 2},
        # independent bubble scenes of uneven sizes tiled into one domain: how training data is generated
        {"name": "bubble_batch_24", "kind": "job", "scene": "batch", "nx": 24, "ny": 0, "nz": 0, "schedule": "fused", "steps": 4},
        # a host that drives plain SPH call by call, as the reference's RunSimpleSPH, and reads every frame back
        {"name": "calls_plain", "kind": "calls", "scene": "plain", "nx": 64, "ny": 48, "nz": 60, "steps": 4},
        # the learned large step: the step with features, the network and its correction
        {"name": "large_step_liquid", "kind": "large", "scene": "liquid", "nx": 128, "ny": 64, "nz": 96, "steps": 4},
        # implicit incompressible SPH with a bounded number of pressure iterations
        {"name": "iisph_dam_32", "kind": "iisph", "scene": "dam_tait", "nx": 32, "ny": 32, "nz": 32, "steps": 1, "iterations": 10},
        # corrector training at the training configuration's batch, and at the default batch of the fit helper
        {"name": "train_65536", "kind": "train", "batch": 65536, "steps": 8},
        {"name": "train_8192", "kind": "train", "batch": 8192, "steps": 8},
        # corrector inference on a ragged number of rows
        {"name": "forward_1000003", "kind": "forward", "rows": 1000003},
    ]


def _spread(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _lattice(rng, lo, hi, most):
    while True:
        n = [_spread(rng, lo, hi) for _ in range(3)]
        if n[0] * n[1] * n[2] <= most:
            return {"nx": n[0], "ny": n[1], "nz": n[2]}


def draw(rng):
    kind = rng.choice(["job", "job", "job", "calls", "large", "iisph", "train", "forward"])
    if kind == "job":
        scene = rng.choice(["dam", "blobs", "liquids", "liquids", "batch"])
        if scene == "batch":
            return {"kind": kind, "scene": scene, "nx": rng.randint(3, 24), "ny": 0, "nz": 0, "schedule": "fused",
                    "steps": rng.randint(1, 4)}
        schedule = rng.choice(["fused", "reference", "projectu"]) if scene == "liquids" else "fused"
        size = _lattice(rng, 12, 48, 40000) if scene == "dam" else _lattice(rng, 14, 128, 500000)
        return {"kind": kind, "scene": scene, **size, "schedule": schedule,
                "steps": rng.randint(1, 3 if schedule == "projectu" else 8),
                "cell_order": rng.choice(["linear", "linear", "morton"])}
    if kind == "calls":
        return {"kind": kind, "scene": "plain", **_lattice(rng, 14, 96, 400000), "steps": rng.randint(1, 5)}
    if kind == "large":
        return {"kind": kind, "scene": "liquid", **_lattice(rng, 16, 128, 700000), "steps": rng.randint(1, 4)}
    if kind == "iisph":
        return {"kind": kind, "scene": "dam_tait", **_lattice(rng, 12, 40, 32768), "steps": 1,
                "iterations": rng.randint(2, 10)}
    if kind == "train":
        return {"kind": kind, "batch": 128 * _spread(rng, 1, 512), "steps": rng.randint(2, 8)}
    return {"kind": "forward", "rows": _spread(rng, 1, 2000000)}


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------

def _scene(case, seed):
    """The scene's parameters and records."""
    kind, size = case["scene"], (case["nx"], case["ny"], case["nz"])
    if kind == "batch":
        sizes = np.random.default_rng(size[0])  # the scenes' sizes go with the case, their particles with the seed
        counts = np.exp(sizes.uniform(np.log(4096), np.log(65536), size[0])).astype(int)
        sc, _ = scenes.tile([scenes.bubble_scene(seed * 1009 + i, int(c)) for i, c in enumerate(counts)])
    elif kind in ("dam", "dam_tait"):
        # a block in the corner of a box twice as long, with a gas sphere under its middle (none under Tait)
        d, h = 0.01, 0.02
        box = tuple(max(n * d * f, 4 * h) for n, f in zip(size, (2.0, 1.5, 1.25)))
        p = scenes.make_params(h=h, d=d, dt=2e-4, box_min=(0.0, 0.0, 0.0), box_max=box, nphase=2, dens=(1000.0, 1.2),
                               visc=(0.2, 0.2), eos=abi.EOS_TAIT if kind == "dam_tait" else abi.EOS_LINEAR,
                               multiphase=0 if kind == "dam_tait" else 1)
        sc = _fill(p, size, d, box, seed)
        if kind == "dam":
            middle = np.array([0.5 * size[0] * d, 0.35 * size[1] * d, 0.5 * size[2] * d], np.float32)
            gas = np.sum((sc.disp["pos"] - middle) ** 2, axis=1) < (0.19 * min(size) * d) ** 2
            _set_phase(sc, gas & (sc.disp["type"] == abi.TYPE_FLUID), 1)
    elif kind == "liquid":
        sc = scenes.rollout_bubbles(seed=seed, lattice=size, liquid_only=True)
    else:  # blobs (gas among them), liquids, plain: the three-phase lattice
        d = 0.005
        box = (2 * size[0] * d, 2 * size[1] * d, size[2] * d)
        blobs = max(8, min(64, size[0] * size[1] * size[2] // 16384))
        sc = scenes.blobs_3phase(seed=seed, lattice=size, box=tuple(max(b, 0.04) for b in box), n_blobs=blobs,
                                 eos=abi.EOS_LINEAR if kind == "blobs" else abi.EOS_TAIT,
                                 multiphase=0 if kind == "plain" else 1)
        if kind != "blobs":  # the third phase a liquid too: the Tait EOS has no use for gas beside liquid
            light = sc.calc["restdens"] == np.float32(sc.params.densArr[2])
            sc.params.densArr[2] = 900.0
            sc.params.massArr[2] = 900.0 * d ** 3
            _set_phase(sc, light & (sc.disp["type"] == abi.TYPE_FLUID), 2)
    if case.get("cell_order") == "morton":
        sc.params.cell_order = abi.CELL_ORDER_MORTON
    return sc


def _fill(p, size, d, box, seed):
    walls = [2 * 2 * (b / d + 8) * (c / d + 8) * 1.3 for b, c in ((box[0], box[1]), (box[0], box[2]), (box[1], box[2]))]
    disp, calc = sphmp.record_arrays(size[0] * size[1] * size[2] + int(sum(walls)) + 4096)
    lo = [0.5 * d] * 3
    n = sphmp.add_fluid_volume(p, disp, calc, 0, lo, [lo[a] + (size[a] - 0.5) * d for a in range(3)], d,
                               jitter=0.1 * d, seed=seed)
    m = sphmp.add_open_box(p, disp, calc, n, (0.0, 0.0, 0.0), box, 1.5 * d)
    p.num = p.maxNum = m
    return scenes.Scene(p, disp[:m].copy(), calc[:m].copy(), n, m - n)


def _set_phase(sc, sel, k):
    sc.calc["restdens"][sel] = sc.params.densArr[k]
    sc.calc["mass"][sel] = sc.params.massArr[k]
    sc.calc["visc"][sel] = sc.params.viscArr[k]


def _pinned(n):
    """Page-locked display and calculation records."""
    return tuple(torch.empty(n * t.itemsize, dtype=torch.uint8, pin_memory=True).numpy().view(t)
                 for t in (abi.display_dtype(), abi.calc_dtype()))


def _network(seed):
    """Parameters and normalisation as a trained corrector has them: weights of order 1/sqrt(width)."""
    rng = np.random.default_rng(seed)
    shift = rng.normal(0.0, 0.3, 48).astype(np.float32)
    scale = rng.uniform(0.5, 2.0, 48).astype(np.float32)
    return learned.init_params(seed), shift, scale, np.array([1e-3, 1e-3, 1e-3, 1e-4], np.float32)


def _rows(n, seed, shift, scale):
    """Raw features whose normalised values are correlated and of order one."""
    g = torch.Generator("cuda")
    g.manual_seed(seed)
    mix = torch.eye(48, device="cuda") + 0.15 * torch.randn(48, 48, device="cuda", generator=g)
    z = torch.randn(n, 48, device="cuda", generator=g) @ mix
    return (z / torch.from_numpy(scale).cuda() + torch.from_numpy(shift).cuda()).contiguous(), z


def _targets(z, seed):
    """A smooth function of the features plus noise: what training fits."""
    g = torch.Generator("cuda")
    g.manual_seed(seed + 1)
    w = torch.randn(48, 4, device="cuda", generator=g) / 7.0
    return (torch.tanh(z @ w) + 0.05 * torch.randn(z.shape[0], 4, device="cuda", generator=g)).contiguous()


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("train", "forward"):
        par, shift, scale, out = _network(seed)
        cor = sphmp.Corrector(case["batch"] if kind == "train" else 0)
        cor.set_params(par)
        cor.set_normalisation(shift, scale, out)
        if kind == "forward":
            x, _ = _rows(case["rows"], seed, shift, scale)
            return {"kind": kind, "cor": cor, "x": x, "y": torch.empty(case["rows"], 4, device="cuda")}
        data = []
        for k in range(case["steps"]):
            x, z = _rows(case["batch"], seed * 31 + k, shift, scale)
            data.append((x, _targets(z, seed)))
        return {"kind": kind, "cor": cor, "data": data}
    sc = _scene(case, seed)
    state = {"kind": kind, "case": dict(case), "ctx": sphmp.Context(sc.params), "in": _pinned(sc.n), "out": _pinned(sc.n)}
    state["in"][0][:] = sc.disp
    state["in"][1][:] = sc.calc
    if kind == "large":
        par, shift, scale, out = _network(seed)
        state["cor"] = sphmp.Corrector(0)
        state["cor"].set_params(par)
        state["cor"].set_normalisation(shift, scale, out)
    return state


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------

def _records(disp, calc):
    names = ("vel", "veleval", "pressure", "dens", "restdens", "visc", "accel", "bornid")
    return {"pos": disp["pos"], "type": disp["type"], **{k: calc[k] for k in names}}


def run(state):
    kind = state["kind"]
    if kind == "forward":
        state["cor"].forward(state["x"], state["y"])
        return {"y": state["y"]}
    if kind == "train":
        for x, t in state["data"]:
            state["cor"].train_step(x, t, LR)
        state["cor"].sync()
        return {"params": state["cor"].get_params()}
    case, ctx = state["case"], state["ctx"]
    ctx.upload_aos(*state["in"])
    ctx.before_first_step()
    more = {}
    if kind == "job":
        ctx.step(case["steps"], SCHEDULES[case["schedule"]])
    elif kind == "large":
        ctx.step_large(8, case["steps"], state["cor"])
    elif kind == "iisph":
        more["iterations"], more["residue"] = ctx.step_iisph(case["steps"], 0.0, case["iterations"])
    else:
        for _ in range(case["steps"]):
            ctx.sort()
            ctx.compute_pressure()
            ctx.compute_force()
            ctx.advance()
            ctx.download_aos(calc=False, out=state["out"])
    ctx.download_aos(out=state["out"])
    if ctx.params.multiphase:
        more["alpha"] = ctx.download_field(abi.F_ALPHA)
    if case.get("schedule") == "projectu":
        more["velxcor"] = ctx.download_field(abi.F_VELXCOR)
    return {**_records(*state["out"]), **more}


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------

def work(case):
    kind = case["kind"]
    if kind in ("train", "forward"):
        macs = sum(a * b for a, b in LAYERS)
        par = 4 * sum(a * b + b for a, b in LAYERS)
        if kind == "forward":
            return {"bytes": case["rows"] * (48 + 4) * 4 + par, "flops": 2.0 * macs * case["rows"]}
        # forward, weight gradients and input gradients (none of the inputs); the parameters and Adam's moments
        per_row = 2.0 * (3 * macs - 48 * 128)
        return {"bytes": case["steps"] * (case["batch"] * (48 + 4) * 4 + 6 * par),
                "flops": case["steps"] * case["batch"] * per_row}
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    if case["scene"] == "batch":
        fluid = nx * (65536 - 4096) / math.log(16.0)  # the mean of the log-uniform counts
        total = fluid * 1.8
    else:
        fluid = nx * ny * nz
        f = {"dam": (2.0, 1.5, 1.25), "dam_tait": (2.0, 1.5, 1.25), "liquid": (1.05, 1.25, 1.05)}.get(case["scene"], (2, 2, 1))
        bx, by, bz = nx * f[0], ny * f[1], nz * f[2]
        total = fluid + 2 * (bx * bz + 2 * by * (bx + bz))  # an open box of two layers
    moved = total * 2 * (32 + 224)  # the records up and down
    pairs = 33.0 * fluid            # neighbours within h = 2 d
    state = 160.0 * total           # five 16-byte fields read and written by a step
    if kind == "iisph":
        flops = pairs * (8 * 15 + 110 + 90 * case["iterations"])
        return {"bytes": moved + total * (160 + 48 * case["iterations"]), "flops": flops}
    if kind == "calls":
        return {"bytes": moved + case["steps"] * (state + 32 * total), "flops": case["steps"] * pairs * 60}
    flops = case["steps"] * pairs * (200 if kind == "job" else 300)
    if kind == "large":
        flops += case["steps"] * total * 2.0 * sum(a * b for a, b in LAYERS)
    return {"bytes": moved + case["steps"] * state, "flops": flops}


# ---------------------------------------------------------------------------
# the same in 64 bits
# ---------------------------------------------------------------------------

def exact(case, seed):
    kind = case["kind"]
    if kind == "large":
        return None  # a step with a 16-bit network inside
    if kind in ("train", "forward"):
        return _exact_network(case, seed)
    sc = _scene(case, seed)
    s = _Exact(sc.params, sc.disp, sc.calc)
    s.sort()
    s.boundary_volume()
    more = {}
    for _ in range(case["steps"]):
        s.sort()
        if kind == "iisph":
            more["iterations"], more["residue"] = [None] * case["steps"], s.step_iisph(case["iterations"])
        else:
            s.step(case.get("schedule", "fused"))
    out = s.records()
    if sc.params.multiphase:
        out["alpha"] = s.alpha
    if case.get("schedule") == "projectu":
        out["velxcor"] = s.xsph
    return {**out, **more}


def _exact_network(case, seed):
    par, shift, scale, _ = _network(seed)
    flat = torch.from_numpy(par).cuda().double().requires_grad_(case["kind"] == "train")
    shift, scale = torch.from_numpy(shift).cuda().double(), torch.from_numpy(scale).cuda().double()

    def net(x):
        h, at = (x.double() - shift) * scale, 0
        for k, (i, o) in enumerate(LAYERS):
            w = flat[at:at + i * o].reshape(o, i)
            b = flat[at + i * o:at + i * o + o]
            at += i * o + o
            h = h @ w.T + b
            h = torch.nn.functional.silu(h) if k < 3 else h
        return h

    if case["kind"] == "forward":
        x, _ = _rows(case["rows"], seed, *_network(seed)[1:3])
        return {"y": torch.cat([net(c) for c in x.split(1 << 18)])}
    m, v = torch.zeros_like(flat), torch.zeros_like(flat)
    for k in range(case["steps"]):
        x, z = _rows(case["batch"], seed * 31 + k, *_network(seed)[1:3])
        loss = (net(x) - _targets(z, seed).double()).square().sum(1).mean()
        g, = torch.autograd.grad(loss, flat)
        with torch.no_grad():
            m = 0.9 * m + 0.1 * g
            v = 0.999 * v + 0.001 * g * g
            flat -= LR * (m / (1 - 0.9 ** (k + 1))) / ((v / (1 - 0.999 ** (k + 1))).sqrt() + 1e-8)
    return {"params": flat.detach()}


class _Exact:
    """The particle state of one scene and its steps: 32-bit state, 64-bit arithmetic."""

    STATE = ("pos", "vel", "vev", "alpha", "rest", "visc", "aprev", "mass", "bound", "bornid", "vol", "dens", "press",
             "acc", "cell")

    def __init__(self, p, disp, calc):
        t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
        d = lambda a: t(a).double()  # noqa: E731
        self.p = p
        self.pos, self.vel, self.vev = d(disp["pos"]), d(calc["vel"]), d(calc["veleval"])
        self.rest, self.visc, self.mass = d(calc["restdens"]), d(calc["visc"]), d(calc["mass"])
        self.bornid, self.bound = t(calc["bornid"]), t(disp["type"]) == abi.TYPE_BOUNDARY
        self.dens, self.press, self.acc = d(calc["dens"]), d(calc["pressure"]), d(calc["accel"])
        self.vol = self.dens.abs()
        n = len(self.rest)
        self.rho_k = [float(np.float32(p.densArr[k])) for k in range(p.nphase)]
        self.nu_k = [float(np.float32(p.viscArr[k])) for k in range(p.nphase)]
        self.alpha = torch.zeros(n, 3, dtype=torch.float64, device="cuda")
        first = torch.zeros(n, dtype=torch.long, device="cuda")
        for k in reversed(range(p.nphase)):
            first[self.rest == self.rho_k[k]] = k
        self.alpha[torch.arange(n, device="cuda"), first] = 1.0
        self.aprev = torch.zeros(n, 3, dtype=torch.float64, device="cuda")
        self.cell = torch.zeros(n, dtype=torch.long, device="cuda")
        self.xsph = torch.zeros(n, 3, dtype=torch.float64, device="cuda")
        self.g = torch.tensor(list(p.gravity), dtype=torch.float64, device="cuda")

    def records(self):
        return {"pos": self.pos, "type": None, "vel": self.vel, "veleval": self.vev,
                "pressure": torch.where(self.bound, 0.0, self.press),
                "dens": torch.where(self.bound, self.vol, self.dens), "restdens": self.rest, "visc": self.visc,
                "accel": self.acc, "bornid": None}

    def sort(self):
        """Stable order by the cell of the reference's grid; out-of-grid particles last."""
        p = self.p
        for k in ("pos", "vel", "vev", "alpha", "rest", "visc", "aprev", "vol"):  # what the arrays hold
            setattr(self, k, getattr(self, k).float().double())
        gmin = torch.tensor(list(p.gridmin), dtype=torch.float32, device="cuda")
        fac = torch.tensor(list(p.gridIdfac), dtype=torch.float32, device="cuda")
        c = torch.trunc((self.pos.float() - gmin) * fac).long()
        rx, ry, rz = list(p.gridres)
        res = torch.tensor([rx, ry, rz], device="cuda")
        self.undef = ((c < 1) | (c >= res - 1)).any(1)
        if p.cell_order == abi.CELL_ORDER_MORTON:
            key = torch.zeros(len(c), dtype=torch.long, device="cuda")
            for b in range(16):
                for k, a in enumerate((0, 2, 1)):
                    key |= ((c[:, a] >> b) & 1) << (3 * b + k)
        else:
            key = (c[:, 1] * rz + c[:, 2]) * rx + c[:, 0]
        key[self.undef] = 1 << 60
        order = torch.sort(key, stable=True).indices
        for k in self.STATE:
            setattr(self, k, getattr(self, k)[order])
        self.undef = self.undef[order]
        self.fluid = ~self.bound & ~self.undef
        self.near = None

    def pairs(self, of, to, radius):
        """(i, j) of the particles i in `of`, j in `to` with 0 < |x_i - x_j| < radius (in metres)."""
        x = self.pos * self.p.simscale
        src, dst = of.nonzero()[:, 0], to.nonzero()[:, 0]
        lo = torch.minimum(x[src].amin(0), x[dst].amin(0)) - radius
        grid = lambda q: torch.floor((x[q] - lo) / radius).long() + 1  # noqa: E731
        cs, cd = grid(src), grid(dst)
        n = torch.maximum(cs.amax(0), cd.amax(0)) + 2
        kd, o = torch.sort((cd[:, 0] * n[1] + cd[:, 1]) * n[2] + cd[:, 2])
        dst = dst[o]
        found = []
        for dx in (-1, 0, 1):
            for dy in (-1, 0, 1):  # the three cells along the last axis are one range
                k = ((cs[:, 0] + dx) * n[1] + cs[:, 1] + dy) * n[2] + cs[:, 2]
                a, b = torch.searchsorted(kd, k - 1), torch.searchsorted(kd, k + 1, right=True)
                for at in range(0, len(src), 1 << 18):
                    a_, m = a[at:at + (1 << 18)], (b - a)[at:at + (1 << 18)]
                    i = torch.repeat_interleave(torch.arange(len(m), device="cuda"), m)
                    first = torch.cumsum(m, 0) - m
                    j = dst[a_[i] + torch.arange(len(i), device="cuda") - first[i]]
                    i = src[i + at]
                    r2 = (x[i] - x[j]).square().sum(1)
                    ok = (r2 < radius * radius) & (r2 > 0)
                    found.append((i[ok], j[ok]))
        return torch.cat([f[0] for f in found]), torch.cat([f[1] for f in found])

    def add(self, i, v):
        return torch.zeros((len(self.rest),) + v.shape[1:], dtype=torch.float64, device="cuda").index_add_(0, i, v)

    def geometry(self):
        """The fluid particles' pairs within h, their distances and the kernel gradient factor."""
        if self.near is None:
            h = float(self.p.smoothradius)
            i, j = self.pairs(self.fluid, ~self.undef, h)
            d = (self.pos[i] - self.pos[j]) * self.p.simscale
            r2 = d.square().sum(1)
            r = r2.sqrt()
            self.near = i, j, d, r2, float(self.p.kspikydiff) * (h - r) ** 2 / r
        return self.near

    def boundary_volume(self):
        h = float(self.p.smoothradius)
        b = self.bound & ~self.undef
        i, j = self.pairs(b, b, h)
        r2 = ((self.pos[i] - self.pos[j]) * self.p.simscale).square().sum(1)
        s = (self.add(i, (h * h - r2) ** 3) + h ** 6) * float(self.p.kpoly6)
        self.vol = torch.where(b, 1.0 / s, self.vol)

    def density(self):
        p, h = self.p, float(self.p.smoothradius)
        i, j, _, r2, _ = self.geometry()
        m = torch.where(self.bound[j], self.rest[i] * self.vol[j], self.mass[j])
        rho = (self.add(i, (h * h - r2) ** 3 * m) + h ** 6 * self.mass) * float(p.kpoly6)
        if p.eos == abi.EOS_LINEAR:
            pr = float(p.eos_stiffness) * (rho - self.rest)
        else:
            pr = 2.5 * self.rest * ((rho / self.rest) ** 7 - 1.0)
        self.dens = torch.where(self.fluid, 1.0 / rho, self.dens)
        self.press = torch.where(self.fluid, pr.clamp(min=0.0), self.press)

    def force(self):
        p, h = self.p, float(self.p.smoothradius)
        i, j, d, r2, g1 = self.geometry()
        f = ~self.bound[j]
        dv = self.vel[i] - self.vel[j]
        di = self.dens[i]
        g = g1 * self.mass[j] * self.dens[j]
        fluid = (-0.5 * g * self.press[j] * di)[:, None] * d + (g * (self.visc[i] + self.visc[j]) * di)[:, None] * dv
        gb = g1 * self.rest[i] * self.vol[j]
        dot = (dv * d).sum(1)
        art = torch.where(dot < 0, dot / (r2 + 0.01 * h * h) * float(p.bvisc) * h / 2 / self.rest[i], 0.0)
        wall = (gb * (art - self.press[i] * di * di))[:, None] * d
        self.acc = torch.where(self.undef[:, None], self.acc, self.add(i, torch.where(f[:, None], fluid, wall)))

    def drift(self):
        p, n = self.p, self.p.nphase
        i, j, d, _, g1 = self.geometry()
        f = ~self.bound[j]
        i, j, d = i[f], j[f], d[f]
        g = g1[f] * self.mass[j] * self.dens[j]
        relax, inv = float(p.mf_relax) / self.visc, 1.0 / self.rest
        a, pr = self.alpha, self.press
        pg = [self.add(i, (g * (a[j, k] * pr[j] - a[i, k] * pr[i]))[:, None] * d) for k in range(n)]
        ag = [self.add(i, (g * (a[j, k] - a[i, k]))[:, None] * d) for k in range(n)]
        mc = [a[:, k] * self.rho_k[k] * inv for k in range(n)]
        mean = sum(mc[k][:, None] * pg[k] for k in range(n))
        cd = [torch.where((a[:, k] > float(np.float32(1e-4)))[:, None], ag[k] / a[:, k:k + 1], 0.0) for k in range(n)]
        cmean = sum(mc[k][:, None] * cd[k] for k in range(n))
        heavy = sum(mc[k] * self.rho_k[k] for k in range(n))
        c, c1, c2 = float(p.mf_cont), float(p.mf_cont1), float(p.mf_cont2)
        self.um = [-c * c2 * relax[:, None] * (pg[k] - mean) + self.aprev * ((self.rho_k[k] - heavy) * relax)[:, None]
                   - c * c1 * float(p.mf_diffusion) * (cd[k] - cmean) for k in range(n)]

    def alpha_change(self):
        p, n = self.p, self.p.nphase
        i, j, d, _, g1 = self.geometry()
        f = ~self.bound[j]
        i, j, d = i[f], j[f], d[f]
        cm = g1[f] * self.mass[j] * self.dens[j]
        dot = ((self.vev[j] - self.vev[i]) * d).sum(1)
        new = self.alpha.clone()
        for k in range(n):
            a, u = self.alpha[:, k], self.um[k]
            flux = ((a[j, None] * u[j] + a[i, None] * u[i]) * d).sum(1)
            ch = self.add(i, -cm * (0.5 * (a[j] + a[i]) * dot + flux)) * float(p.dt)
            new[:, k] = torch.where(self.fluid, a + ch.clamp(min=-0.99), a)
        return new

    def correct(self, new):
        p, n = self.p, self.p.nphase
        old = self.alpha
        a = new.clone()
        a[:, :n] = a[:, :n].clamp(min=0.0)
        s = a[:, :n].sum(1, keepdim=True)
        hot = torch.zeros_like(a).scatter_(1, old[:, :n].argmax(1, keepdim=True), 1.0)
        a = torch.where(s > 0, a / torch.where(s > 0, s, 1.0), hot)
        f = self.fluid
        self.before = old
        self.alpha = torch.where(f[:, None], a, old)
        self.rest = torch.where(f, sum(a[:, k] * self.rho_k[k] for k in range(n)), self.rest)
        self.visc = torch.where(f, sum(a[:, k] * self.nu_k[k] for k in range(n)), self.visc)

    def force_projectu(self):
        p, h, n = self.p, float(self.p.smoothradius), self.p.nphase
        i, j, d, r2, g1 = self.geometry()
        f = ~self.bound[j]
        dv = self.vev[i] - self.vev[j]
        di = self.dens[i]
        dj = torch.where(f, self.dens[j], self.vol[j])
        g = g1 * self.mass[j] * dj
        fl = (-0.5 * g * (self.press[i] + self.press[j]) * di)[:, None] * d
        fl = fl + (g * (self.visc[i] + self.visc[j]) * di)[:, None] * dv
        for k in range(n):
            for q in (j, i):
                u, a = self.um[k][q], self.before[q, k]
                fl = fl + (g * (u * d).sum(1) * a * self.rho_k[k] * di)[:, None] * u
        gb = g1 * self.rest[i] * self.mass[j] / self.rest[j]
        dot = (dv * d).sum(1)
        art = dot / (r2 + 0.01 * (h / float(p.simscale)) ** 2) * h * (self.visc[i] + self.visc[j]) * di
        art = torch.where(dot < 0, -gb * art * float(p.mf_visc_factor), 0.0)
        wall = (art - gb * self.press[i] * di * di * float(p.mf_omega))[:, None] * d
        self.acc = torch.where(self.undef[:, None], self.acc, self.add(i, torch.where(f[:, None], fl, wall)))
        w = (h * h - r2) ** 3 * self.mass[j] * (2.0 / (1.0 / dj + 1.0 / di)) * float(p.kpoly6) * 0.5
        self.xsph = self.add(i, -w[:, None] * dv)

    def advance(self):
        p, f = self.p, self.fluid[:, None]
        dt = float(p.dt)
        a = self.acc + self.g
        v = self.vel + a * dt
        park = (self.undef & ~self.bound)[:, None]
        self.pos = torch.where(f, self.pos + v * dt / float(p.simscale), torch.where(park, -1000.0, self.pos))
        self.vev = torch.where(f, 0.5 * (self.vel + v), self.vev)
        self.vel = torch.where(f, v, torch.where(park, 0.0, self.vel))
        self.aprev = torch.where(f, self.g - a, self.aprev)

    def step(self, schedule):
        self.density()
        if not self.p.multiphase:
            self.force()
        elif schedule == "fused":  # the force before the correction
            self.drift()
            self.force()
            self.correct(self.alpha_change())
        else:
            self.drift()
            self.correct(self.alpha_change())
            self.force() if schedule == "reference" else self.force_projectu()
        self.advance()

    def nabla(self, d):
        """The gradient of the cubic spline of support 2h."""
        h = float(self.p.smoothradius)
        r = d.square().sum(1).sqrt()
        q = r / h
        inner, outer = -3.0 * q + 2.25 * q * q, -0.75 * (2.0 - q) ** 2
        return (torch.where(q > 1, outer, inner) / h / r * float(self.p.kspline))[:, None] * d

    def step_iisph(self, iterations):
        """One implicit step with a fixed number of pressure iterations; returns its two residues."""
        p, h, ss, dt = self.p, float(self.p.smoothradius), float(self.p.simscale), float(self.p.dt)
        f = self.fluid
        i, j = self.pairs(f, ~self.undef, 2 * h)
        d = (self.pos[i] - self.pos[j]) * ss
        q = d.square().sum(1).sqrt() / h
        w = torch.where(q > 1, 0.25 * (2.0 - q) ** 3, 1.0 - 1.5 * q * q + 0.75 * q ** 3) * float(p.kspline)
        m = torch.where(self.bound[j], self.rest[i] * self.vol[j], self.mass[j])
        rho = torch.where(f, self.add(i, w * m) + float(p.kspline) * self.mass, self.dens)
        b = self.bound[j]
        i, j, d = i[b], j[b], d[b]
        dv = self.vel[i] - self.vel[j]
        dot = (dv * d).sum(1)
        art = dot / (d.square().sum(1) + 0.01 * h * h) * float(p.bvisc) * h / 2 / self.rest[i]
        art = torch.where(dot < 0, self.rest[i] * self.vol[j] * art, 0.0)
        adv = self.add(i, art[:, None] * self.nabla(d)) + self.g
        vev = torch.where(f[:, None], self.vel + adv * dt, self.vev)
        i, j = self.pairs(f, f, h)
        d = (self.pos[i] - self.pos[j]) * ss
        nw, mi, mj = self.nabla(d), self.mass[i], self.mass[j]
        dii = self.add(i, -nw * mj[:, None]) / (rho * rho)[:, None] * dt * dt
        radv = rho + self.add(i, ((vev[i] - vev[j]) * nw).sum(1) * mj * dt)
        dji = nw * (mi / (rho[i] * rho[i]) * dt * dt)[:, None]
        aii = self.add(i, ((dii[i] - dji) * nw).sum(1) * mj)
        pl = 0.5 * self.press
        for _ in range(iterations):
            dp = self.add(i, -nw * (pl[j] * mj / (rho[j] * rho[j]))[:, None]) * dt * dt
            t = dp[i] - dii[j] * pl[j, None] - (dp[j] - dji * pl[i, None])
            ut = self.add(i, mj * (t * nw).sum(1))
            res = torch.where(f, radv + ut + aii * pl - self.rest, 0.0)
            acc = (dii * pl[:, None] + dp) / dt / dt
            new = torch.where(aii.abs() < 1e-5, pl, 0.9 * pl + 0.1 / aii * (self.rest - radv - ut))
            pl = torch.where(f, new, pl)
        self.acc = torch.where(f[:, None], acc, self.acc)
        self.press = torch.where(f, pl, self.press)
        self.dens = rho
        self.vel = torch.where(f[:, None], vev + self.acc * dt, self.vel)
        self.vev = vev
        self.pos = torch.where(f[:, None], self.pos + self.vel * dt / ss, self.pos)
        return float(res.sum()) / len(res), float(res.abs().sum()) / int(f.sum())
