"""Workloads that the library's speed is measured on, each through its public
entry points (the C ABI and the Python host layer over it).

Five kinds of work, as programs that use the library have it do them:

  steps      a solver run's inner loop: the timesteps between two reads of the
             state, then the state (positions and velocities by particle id)
             copied out to pinned host memory, as for a state file.
  roundtrip  the host program that keeps the state itself: uploads it, calls
             the timestep one step at a time and reads the counters after each
             (System::step and the sampler call of the reference's main), and
             downloads it.
  fields     an ensemble of porous geometries advanced together, with the
             per-voxel sums of every geometry accumulated every ten steps
             (steady fields, the warm start's training data).
  conv       one periodic 3x3x3 convolution layer of the warm-start network,
             forward with bias and ReLU, or (conv_bwd) its backward: weight,
             bias and masked input gradient.
  unet       the whole network's inference on a batch of boxes, or
             (unet_train) a training step: forward, backward, Adam.

Sizes are the repository's own workloads (master_b200/workloads.py, the
network's layers, the batch of its training) or, drawn, anything between.
"""
from __future__ import annotations

import ctypes as C
import functools
import math
import random

import numpy as np
import torch

from master_b200 import capi, fields, surrogate
from master_b200.system import T0_TEMP, Context, Geometry, System
from master_b200.workloads import Workload, simulators_per_cell_weight

CHANNELS = (16, 32, 48, 64, 96)
DENSITY = 2.5e24
VOXEL_UM = 0.1


# ---- cases -----------------------------------------------------------------

def listed():
    return [
        # a small porous sample, 3.9e5 particles: the steps between two reads
        # of the state at the default statistics interval (launches and
        # latencies count most)
        dict(name="steps_64", kind="steps", edge=64, cells=32, porosity=0.6, radius=4.0, per_cell=20.0, steps=100,
             precision="split", wall=0, interval=0),
        # the same in the reference's own fp64 arithmetic
        dict(name="steps_64_fp64", kind="steps", edge=64, cells=32, porosity=0.6, radius=4.0, per_cell=20.0, steps=40,
             precision="fp64", wall=0, interval=0),
        # a medium sample, 3.9e6 particles, sampled every ten steps, with
        # Cercignani-Lampis walls; the sampler's moments and profiles are read
        # with the state
        dict(name="sampled_128", kind="steps", edge=128, cells=64, porosity=0.5, radius=6.0, per_cell=30.0, steps=100,
             precision="split", wall=2, interval=10),
        # the headline run: 3.15e7 particles
        dict(name="steps_256", kind="steps", edge=256, cells=128, porosity=0.5, radius=6.0, per_cell=30.0, steps=200,
             precision="split", wall=0, interval=0),
        # the drop-in use: state up, twenty calls of one step each with the
        # counters read after it, state down
        dict(name="roundtrip_128", kind="roundtrip", edge=128, cells=64, porosity=0.5, radius=6.0, per_cell=30.0,
             steps=20),
        # sixteen geometries of uneven size in one context, fields accumulated
        dict(name="fields_16_uneven", kind="fields", systems=16, geometry_seed=3, edge_max=128, per_cell=30.0,
             steps=50, every=10),
        # the coarsest level of one box: the smallest layer call
        dict(name="conv_16_64to64", kind="conv", S=16, batch=1, cin=64, cout=64),
        # the finest level's widest layer (decoder, 48 -> 16), batch of training
        dict(name="conv_64_48to16", kind="conv", S=64, batch=8, cin=48, cout=16),
        # the backward of the middle level's widest layer (decoder, 96 -> 32)
        dict(name="conv_bwd_32_96to32", kind="conv_bwd", S=32, batch=8, cin=96, cout=32),
        # the backward of a finest-level layer
        dict(name="conv_bwd_64_16to16", kind="conv_bwd", S=64, batch=8, cin=16, cout=16),
        # inference on a batch of boxes, and a training step on it
        dict(name="unet_64", kind="unet", S=64, batch=8),
        dict(name="unet_train_64", kind="unet_train", S=64, batch=8),
    ]


def _log(rng, a, b):
    return math.exp(rng.uniform(math.log(a), math.log(b)))


def draw(rng: random.Random):
    kind = rng.choice(["steps", "steps", "steps", "roundtrip", "fields", "conv", "conv", "conv_bwd", "conv_bwd",
                       "unet", "unet_train"])
    if kind in ("steps", "roundtrip"):
        vpc = rng.choice([2, 2, 2, 4])                  # voxels per cell and axis
        edge = vpc * round(_log(rng, 24, 160) / vpc)
        c = dict(kind=kind, edge=edge, cells=edge // vpc, porosity=round(rng.uniform(0.4, 0.8), 3),
                 radius=round(rng.uniform(3.0, 8.0), 2),
                 per_cell=round(_log(rng, 10, 40) if vpc == 2 else _log(rng, 30, 80), 2))
        if kind == "roundtrip":
            c["steps"] = rng.randint(5, 40)
            return c
        c["precision"] = rng.choice(["split", "split", "split", "fp64"])
        c["wall"] = rng.choice([0, 0, 1, 2])
        c["interval"] = rng.choice([0, 0, 10, 25])
        c["steps"] = round(_log(rng, 40, 200)) if c["precision"] == "split" else rng.randint(20, 50)
        return c
    if kind == "fields":
        return dict(kind=kind, systems=rng.randint(2, 24), geometry_seed=rng.randrange(1, 10 ** 6),
                    edge_max=rng.choice([48, 64, 96]), per_cell=round(_log(rng, 15, 60), 2), steps=50, every=10)
    if kind in ("conv", "conv_bwd"):
        S = rng.choice([8, 16, 32, 64])
        most = 8 * 64 ** 3 // S ** 3
        return dict(kind=kind, S=S, batch=round(_log(rng, 1, min(most, 64))), cin=rng.choice(CHANNELS),
                    cout=rng.choice(CHANNELS))
    S = rng.choice([16, 32, 64])
    batch = round(_log(rng, 1, min(8 * 64 ** 3 // S ** 3, 48)))
    # (the coarsest level's voxels come in multiples of 128)
    return dict(kind=kind, S=S, batch=batch + batch % 2 if S == 16 else batch)


# ---- DSMC ------------------------------------------------------------------

def _workload(c) -> Workload:
    # (F_N = n V_cell / per_cell as the benchmark's workloads; the 64^3 one's 1000 at 20 per cell)
    return Workload("case", n=c["edge"], radius_voxels=c["radius"], porosity=c["porosity"], geometry_seed=1,
                    cells=c["cells"],
                    atoms_per_molecule=simulators_per_cell_weight(DENSITY, VOXEL_UM, c["edge"] // c["cells"],
                                                                  c["per_cell"]))


@functools.lru_cache(maxsize=24)
def _pack(n, radius, porosity, seed) -> Geometry:
    return Geometry.packed_spheres(n, radius, wanted_porosity=porosity, seed=seed)


def _pinned(n):
    return torch.empty((n, 3), dtype=torch.float64).pin_memory()


_D = C.POINTER(C.c_double)


def _dp(t):
    return C.cast(t.data_ptr(), _D)


class _Dsmc:
    """One system with the host buffers of a program that reads its state."""

    def __init__(self, c, seed):
        w = _workload(c)
        self.case = c
        interval = c.get("interval", 0)
        s = w.settings(rng_seed=1 + seed, statistics_interval=interval or 10 ** 9)
        s.surface_model = c.get("wall", 0)
        if s.surface_model == 2:
            s.alpha_n, s.alpha_t = 0.8, 0.8
        precision = capi.PREC_FP64 if c.get("precision") == "fp64" else capi.PREC_SPLIT32
        self.system = System(s, _pack(w.n, w.radius_voxels, w.porosity, w.geometry_seed),
                             context=Context(0, precision))
        self.n = self.system.num_molecules
        self.r, self.v = _pinned(self.n), _pinned(self.n)
        self.counters = np.zeros(8, np.int64)
        if c["kind"] == "roundtrip":
            self.r0, self.v0 = self.host_state(s, seed)

    def host_state(self, s, seed):
        """A host program's own state: uniform in the empty voxels (a hair
        inside them), Maxwellian velocities."""
        g = _gen(seed)
        vox = torch.from_numpy(self.system.geometry.voxels).cuda()
        empty = (vox.reshape(-1) == 0).nonzero()[:, 0]
        at = empty[torch.randint(len(empty), (self.n,), generator=g, device="cuda")]
        n = self.case["edge"]
        ijk = torch.stack([at // (n * n), at // n % n, at % n], 1).double()
        u = torch.rand((self.n, 3), generator=g, device="cuda", dtype=torch.float64)
        r = (ijk + 1e-4 + (1.0 - 2e-4) * u) * VOXEL_UM
        v = torch.randn((self.n, 3), generator=g, device="cuda", dtype=torch.float64)
        v *= math.sqrt(s.temperature / T0_TEMP / s.mass)
        return r.cpu().pin_memory(), v.cpu().pin_memory()

    def read_counters(self):
        ctx = self.system.ctx
        ctx.check(ctx.lib.dsmc_counters_get(ctx.handle, self.system.id,
                                            self.counters.ctypes.data_as(C.POINTER(C.c_int64))))

    def download(self):
        ctx = self.system.ctx
        got = C.c_int64()
        ctx.check(ctx.lib.dsmc_particles_get(ctx.handle, self.system.id, self.n, _dp(self.r), _dp(self.v), None,
                                             C.byref(got)))

    def run_steps(self):
        c = self.case
        self.system.step(c["steps"])
        self.download()
        self.read_counters()
        out = {"r": self.r, "v": self.v, "counters": self.counters}
        if c["interval"]:
            cells = self.system.cells()
            out.update(moments=cells["moments"], count=cells["count"], rest=cells["rest"],
                       profiles=self.system.profile_sums())
        return out

    def run_roundtrip(self):
        ctx = self.system.ctx
        ctx.check(ctx.lib.dsmc_particles_set(ctx.handle, self.system.id, self.n, _dp(self.r0), _dp(self.v0)))
        for _ in range(self.case["steps"]):
            self.system.step(1)
            self.read_counters()
        self.download()
        return {"r": self.r, "v": self.v, "counters": self.counters}


def _specs(c):
    rng = np.random.default_rng(c["geometry_seed"])
    specs = fields.random_specs(c["systems"], 32, seed=c["geometry_seed"], per_cell=c["per_cell"])
    edges = [e for e in (32, 48, 64, 96, 128) if e <= c["edge_max"]]
    for sp in specs:
        sp.n = int(rng.choice(edges))
    return specs


class _Fields:
    def __init__(self, c, seed):
        self.case = c
        specs = _specs(c)
        geoms = [_pack(sp.n, sp.radius_voxels, sp.porosity, sp.seed) for sp in specs]
        self.ens = fields.Ensemble(specs, rng_seed=1 + seed, geoms=geoms)
        self.sums = [torch.zeros((sp.n ** 3, 4), dtype=torch.float32, device="cuda") for sp in specs]
        torch.cuda.synchronize()  # zeroed before the context's stream adds to them

    def run(self):
        ctx = self.ens.ctx
        for _ in range(self.case["steps"] // self.case["every"]):
            ctx.step(self.case["every"])
            for S, f in zip(self.ens.systems, self.sums):
                ctx.check(ctx.lib.dsmc_field_accumulate(ctx.handle, S.id, C.c_void_p(f.data_ptr()), 1))
        ctx.sync()
        return self.sums


# ---- the network -----------------------------------------------------------

def _stream():
    return C.c_void_p(torch.cuda.current_stream().cuda_stream)


def _vp(t):
    return C.c_void_p(t.data_ptr() if t is not None else 0)


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(1000003 * (seed + 1))


class _Conv:
    """A layer's tensors: activations after a ReLU, He-normal weights, and for
    the backward an output gradient masked by its ReLU."""

    def __init__(self, c, seed):
        self.case = c
        g = _gen(seed)
        B, S, ci, co = c["batch"], c["S"], c["cin"], c["cout"]

        def randn(*shape):
            return torch.randn(shape, generator=g, device="cuda")
        self.x = torch.relu(randn(B, S, S, S, ci)).to(torch.bfloat16)
        self.w = randn(co, 27, ci) * math.sqrt(2.0 / (27 * ci))
        self.bias = 0.1 * randn(co)
        self.wf = torch.empty((co, 27, ci), dtype=torch.bfloat16, device="cuda")
        self.wd = torch.empty((ci, 27, co), dtype=torch.bfloat16, device="cuda")
        capi.check(capi.load().dsmc_sg_pack_weights(_stream(), _vp(self.w), co, ci, _vp(self.wf), _vp(self.wd)))
        if c["kind"] == "conv":
            self.y = torch.empty((B, S, S, S, co), dtype=torch.bfloat16, device="cuda")
        else:
            dy = randn(B, S, S, S, co)
            self.dy = (1e-3 * dy * (torch.rand(dy.shape, generator=g, device="cuda") < 0.5)).to(torch.bfloat16)
            self.dx = torch.empty_like(self.x)
            self.dw = torch.zeros((co, 27, ci), device="cuda")
            self.db = torch.zeros(co, device="cuda")

    def run_forward(self):
        c, lib = self.case, capi.load()
        capi.check(lib.dsmc_sg_conv3(_stream(), c["batch"], c["S"], _vp(self.x), c["cin"], 0, c["cin"], _vp(self.wf),
                                     _vp(self.bias), c["cout"], _vp(self.y), c["cout"], 0, 1, None, 0, 0))
        return self.y

    def run_backward(self):
        c, lib, s = self.case, capi.load(), _stream()
        B, S, ci, co = c["batch"], c["S"], c["cin"], c["cout"]
        self.dw.zero_()
        self.db.zero_()
        capi.check(lib.dsmc_sg_conv3_wgrad(s, B, S, _vp(self.dy), co, 0, co, _vp(self.x), ci, 0, ci, _vp(self.dw)))
        capi.check(lib.dsmc_sg_bias_grad(s, B, S, _vp(self.dy), co, 0, co, _vp(self.db)))
        capi.check(lib.dsmc_sg_conv3(s, B, S, _vp(self.dy), co, 0, co, _vp(self.wd), None, ci, _vp(self.dx), ci, 0, 0,
                                     _vp(self.x), ci, 0))
        return {"dw": self.dw, "db": self.db, "dx": self.dx}


def _trained() -> np.ndarray:
    """The committed weights, flat."""
    from pathlib import Path
    with np.load(Path(surrogate.__file__).parent / "weights" / "surrogate_64.npz") as z:
        return np.ascontiguousarray(z["params"], np.float32)


class _Unet:
    """The trained network and a batch of porous masks (thresholded smooth
    noise of pore sizes like the sphere packs'), with target fields for the
    training step."""

    def __init__(self, c, seed):
        self.case = c
        g = _gen(seed)
        B, S = c["batch"], c["S"]
        self.net = surrogate.UNet(0, params=_trained())
        noise = torch.randn((B, 1, S, S, S), generator=g, device="cuda")
        for _ in range(2):
            noise = torch.nn.functional.avg_pool3d(torch.nn.functional.pad(noise, (2,) * 6, mode="circular"), 5, 1)
        noise = noise.reshape(B, -1)
        por = 0.4 + 0.4 * torch.rand((B, 1), generator=g, device="cuda")
        order = noise.argsort(dim=1).argsort(dim=1)
        self.solid = (order.float() >= por * S ** 3).to(torch.uint8).reshape(B, S, S, S).contiguous()
        self.feature = 2.0 * torch.rand(B, generator=g, device="cuda") - 1.0
        if c["kind"] == "unet_train":
            self.valid = (self.solid == 0).to(torch.uint8)
            t = torch.randn((B, S, S, S, 4), generator=g, device="cuda")
            t[..., 0] = 1.0 + 0.3 * t[..., 0]
            t[..., 1] += 1.0
            self.target = (t * self.valid[..., None]).contiguous()
            self.cw = torch.tensor([1.0, 4.0, 1.0, 1.0], device="cuda")

    def run(self):
        out = self.net.forward(self.solid, self.feature)
        if self.case["kind"] == "unet":
            return out
        self.net.loss_acc.zero_()
        self.net.backward(self.target, self.valid, self.cw, flux_weight=100.0)
        self.net.adam(lr=5e-5)
        return {"grad": self.net.g, "m": self.net.m, "v": self.net.v, "loss": self.net.loss_acc, "out": out}


# ---- the interface ---------------------------------------------------------

def prepare(case, seed):
    kind = case["kind"]
    if kind in ("steps", "roundtrip"):
        return _Dsmc(case, seed)
    if kind == "fields":
        return _Fields(case, seed)
    if kind in ("conv", "conv_bwd"):
        return _Conv(case, seed)
    return _Unet(case, seed)


def run(state):
    kind = state.case["kind"]
    if kind == "steps":
        return state.run_steps()
    if kind == "roundtrip":
        return state.run_roundtrip()
    if kind == "conv":
        return state.run_forward()
    if kind == "conv_bwd":
        return state.run_backward()
    return state.run()


def _particles(c) -> float:
    return c["per_cell"] * c["porosity"] * c["cells"] ** 3


def work(case):
    """Each particle record read and written once per step (32 bytes, 64 in
    fp64, each way); the uploaded and downloaded state 48 bytes; a field's
    sums read the records once more.  A network: its inputs and outputs, and
    two operations per multiply-add of its convolutions."""
    c = case
    kind = c["kind"]
    if kind in ("steps", "roundtrip"):
        n = _particles(c)
        rec = 128.0 if c.get("precision") == "fp64" else 64.0
        by = n * (rec * c["steps"] + 48.0)
        if kind == "roundtrip":
            by += 48.0 * n
        elif c["interval"]:
            by += n * rec / 2 * (c["steps"] // c["interval"])
        return {"bytes": by, "flops": 20.0 * n * c["steps"]}
    if kind == "fields":
        n = sum(sp.per_cell * sp.porosity * (sp.n // 2) ** 3 for sp in _specs(c))
        v = sum(sp.n ** 3 for sp in _specs(c))
        k = c["steps"] // c["every"]
        return {"bytes": 64.0 * n * c["steps"] + k * (32.0 * n + 32.0 * v), "flops": 20.0 * n * c["steps"]}
    V = c["batch"] * c["S"] ** 3
    if kind in ("conv", "conv_bwd"):
        ci, co = c["cin"], c["cout"]
        f = 2.0 * V * 27 * ci * co
        if kind == "conv":
            return {"bytes": 2.0 * (V * (ci + co) + 27 * ci * co), "flops": f}
        return {"bytes": 2.0 * V * (2 * ci + co) + 6.0 * 27 * ci * co, "flops": 2 * f}
    f = sum(2.0 * (V >> (3 * lev)) * 27 * ci * co for _, ci, co, lev in surrogate.LAYERS)
    if kind == "unet":
        return {"bytes": 17.0 * V + 4.0 * 359812, "flops": f}
    first = 2.0 * V * 27 * 16 * 16  # the first layer has no input gradient
    return {"bytes": 34.0 * V + 32.0 * 359812, "flops": 3 * f - first}


# ---- 64-bit values of the network's cases ----------------------------------
# A particle run has none: its trajectories are chaotic, so the only exact
# answer is the run itself, and its outputs are compared as they are.

class _Conv64(torch.autograd.Function):
    """y[b, v, co] = sum_t x[b, v + off(t), ci] w[co, t, ci], periodic."""

    @staticmethod
    def _off(t):
        return (t // 9 - 1, (t // 3) % 3 - 1, t % 3 - 1)

    @staticmethod
    def forward(ctx, x, w):
        ctx.save_for_backward(x, w)
        y = x.new_zeros(x.shape[:-1] + (w.shape[0],))
        for t in range(27):
            d = _Conv64._off(t)
            y += torch.roll(x, (-d[0], -d[1], -d[2]), (1, 2, 3)) @ w[:, t].T
        return y

    @staticmethod
    def backward(ctx, dy):
        x, w = ctx.saved_tensors
        dx, dw = torch.zeros_like(x), torch.zeros_like(w)
        for t in range(27):
            d = _Conv64._off(t)
            back = torch.roll(dy, d, (1, 2, 3))  # dy[v - off]
            dx += back @ w[:, t]
            dw[:, t] = back.reshape(-1, w.shape[0]).T @ x.reshape(-1, x.shape[-1])
        return dx, dw


def _pool64(x):
    B, S, c = x.shape[0], x.shape[1], x.shape[-1]
    return x.reshape(B, S // 2, 2, S // 2, 2, S // 2, 2, c).mean(dim=(2, 4, 6))


def _up64(x):
    return x.repeat_interleave(2, 1).repeat_interleave(2, 2).repeat_interleave(2, 3)


def _forward64(p, layout, solid, feature):
    def par(key):
        o, sh = layout[key]
        return p[o:o + int(np.prod(sh))].reshape(sh)

    def conv(x, name):
        return torch.relu(_Conv64.apply(x, par(name + ".w")) + par(name + ".b"))
    x = torch.zeros(solid.shape + (16,), dtype=torch.float64, device="cuda")
    x[..., 0] = (solid == 0).double()
    x[..., 1] = feature.double().reshape(-1, 1, 1, 1)
    s1 = conv(conv(x, "c1a"), "c1b")
    s2 = conv(conv(_pool64(s1), "c2a"), "c2b")
    b3 = conv(conv(_pool64(s2), "c3a"), "c3b")
    e2 = conv(conv(torch.cat([_up64(b3), s2], -1), "c2c"), "c2d")
    e1 = conv(conv(torch.cat([_up64(e2), s1], -1), "c1c"), "c1d")
    return e1 @ par("head.w").T + par("head.b")


def exact(case, seed):
    kind = case["kind"]
    if kind not in ("conv", "conv_bwd", "unet", "unet_train"):
        return None
    s = prepare(case, seed)
    if kind == "conv":
        y = torch.relu(_Conv64.apply(s.x.double(), s.w.double()) + s.bias.double())
        return y
    if kind == "conv_bwd":
        x, w = s.x.double().requires_grad_(True), s.w.double().requires_grad_(True)
        _Conv64.apply(x, w).backward(s.dy.double())
        return {"dw": w.grad, "db": s.dy.double().sum(dim=(0, 1, 2, 3)), "dx": x.grad * (s.x.double() > 0)}
    p = s.net.p.double().requires_grad_(kind == "unet_train")
    if kind == "unet":
        with torch.no_grad():
            return _forward64(p, s.net.layout, s.solid, s.feature)
    out = _forward64(p, s.net.layout, s.solid, s.feature)
    valid, tgt = s.valid.double(), s.target.double()
    diff = (out - tgt) * valid[..., None]
    B = s.case["batch"]
    loss = (diff ** 2 * s.cw.double()).sum() / max(1.0, float(valid.sum()))
    nb = valid.reshape(B, -1).sum(1).clamp(min=1.0)
    mean = diff[..., 1].reshape(B, -1).sum(1) / nb
    loss = loss + 100.0 * (mean ** 2).sum() / B
    loss.backward()
    g = p.grad
    return {"grad": g, "m": 0.1 * g, "v": None, "loss": loss.detach().reshape(1), "out": out.detach()}
