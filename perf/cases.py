"""The work that a user of this framework has it do, as cases that can be timed.

Three kinds of case, each through the public Python entry points (lbmc.py over
the C ABI of include/lbmc.h):

* ``step``   one domain: ``Engine.iterate`` for a number of time steps, the last
             of which stores rho and u and reduces the FP64 sums, then the
             fields are fetched.  This is what the run-control loop does between
             two outputs; the handle is kept between passes, as a program keeps
             it, so a pass goes on from where the last one stopped.
* ``sweep``  many uneven 2-D domains to a steady state or a step cap:
             ``Batch`` is built, run and read (a batch that reached its cap is
             finished, so a program builds a new one for new geometries).
* ``train``  the learned subgrid closure's network: loss and gradient of the
             whole set, then mini-batch Adam (``Mlp.gradients``, ``Mlp.train``).

The flows are those of the repository's own configurations: the Poiseuille
channel, the porous sphere pack with pressure faces, the Taylor-Green vortex
with Smagorinsky, the forced box with the learned closure, and random circular
obstacles with partially solid edges.  Fields are handed back as a program
keeps them, in the precision that the engine computes in (float32 snapshots,
float64 for FP64 storage).
"""
from __future__ import annotations

import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "lbm-c_b200"))

import lbmc  # noqa: E402

DEV = "cuda"
F64 = torch.float64

CHANNEL_TAU, CHANNEL_G = 0.8, 1e-6
POROUS_TAU, RHO_IN, RHO_OUT = 0.7, 1.001, 0.999
POROUS_RATES = (0.0, 1.19, 1.19, 0.0, 1.2, 0.0, 1.2, 0.0, 1.2) + (1.0 / POROUS_TAU,) * 5 + (1.2,)
VORTEX_U0, VORTEX_RE, C_SMAG = 0.05, 1600.0, 0.1
BOX_TAU, BOX_URMS, BOX_AMP, BOX_NU_T = 0.5025, 0.03, 2e-6, 2e-3
SWEEP_TAU, SWEEP_G, SWEEP_TOL, SWEEP_CHECK = 1.0, 1e-6, 1e-9, 100
TRAIN_LR = 2e-3


def _step(name, flow, lx, ly, lz, storage, streaming, steps, passes=0):
    return dict(name=name, kind="step", flow=flow, lx=lx, ly=ly, lz=lz, storage=storage,
                streaming=streaming, steps=steps, passes=passes)


def listed():
    return [
        # The smallest call: the 2-D Poiseuille channel between two steady-state checks, in the
        # layout that the run-control program takes.
        _step("channel_128x64", "channel", 128, 64, 1, "f32", "aa", 100),
        # A test-sized porous sample that stays in the L2 cache.
        _step("porous_64", "porous", 64, 64, 64, "f32", "aa", 100),
        # A porous sample cut from a scan: no side a multiple of anything, the layout that
        # make_config takes when nothing is said.
        _step("porous_ragged", "porous", 101, 75, 93, "f32", "shift", 100),
        # The headline benchmark: FP32 storage, and FP16 with stochastic rounding.
        _step("porous_256", "porous", 256, 256, 256, "f32", "aa", 500),
        _step("porous_256_f16sr", "porous", 256, 256, 256, "f16sr", "aa", 500),
        # Decaying turbulence with the subgrid model, half the memory per node.
        _step("vortex_256_bf16", "vortex", 256, 256, 256, "bf16", "aa", 200),
        # The FP64 run that the accuracy studies are measured against.
        _step("vortex_160_f64", "vortex", 160, 160, 160, "f64", "aa", 100),
        # A coarse box with the learned closure, as the closure study runs it.
        _step("closure_64", "box", 64, 64, 64, "f32", "shift", 100, passes=1),
        # One large 2-D porous plane (partially solid edges, body force), stepped alone.
        _step("obstacles_1500x1100", "obstacles", 1500, 1100, 1, "f32", "shift", 200),
        # The permeability sweep in both of its storages, side lengths log-uniform in 32..512.
        dict(name="sweep_f32", kind="sweep", domains=192, storage="f32", cap=3000),
        dict(name="sweep_f16", kind="sweep", domains=192, storage="f16", cap=3000),
        # Training the closure as the study does (its batch size and epochs), on three sixteenths
        # of its samples.
        dict(name="train_196608", kind="train", samples=3 << 16, batch=4096, epochs=8),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    flow = rng.choice(["channel", "porous", "porous", "porous", "vortex", "box", "obstacles", "sweep", "train"])
    streaming = rng.choice(["aa", "shift"])
    if flow == "channel":
        c = _step("", flow, _log_int(rng, 48, 600), _log_int(rng, 24, 200), 1, rng.choice(["f32", "f32", "f64"]),
                  streaming, rng.randrange(50, 200))
    elif flow == "porous":
        side = _log_int(rng, 48, 220)
        lx = side // 64 * 64 if side >= 64 and rng.random() < 0.5 else side
        c = _step("", flow, lx, max(40, int(side * rng.uniform(0.7, 1.2))), max(40, int(side * rng.uniform(0.7, 1.2))),
                  rng.choice(["f32", "f32", "f16sr", "f16", "bf16", "f64"]), streaming, rng.randrange(50, 250))
    elif flow == "vortex":
        side = _log_int(rng, 48, 200)
        c = _step("", flow, side, side, side, rng.choice(["f32", "f16", "bf16", "f64"]), streaming,
                  rng.randrange(50, 150))
    elif flow == "box":
        side = _log_int(rng, 32, 128)
        c = _step("", flow, side, side, side, "f32", streaming, rng.randrange(50, 150), passes=rng.choice([1, 2]))
    elif flow == "obstacles":
        c = _step("", flow, _log_int(rng, 200, 2500), _log_int(rng, 200, 2000), 1, rng.choice(["f32", "f16"]),
                  streaming, rng.randrange(100, 250))
    elif flow == "sweep":
        c = dict(kind="sweep", domains=_log_int(rng, 24, 180), storage=rng.choice(["f32", "f16", "bf16"]),
                 cap=100 * rng.randrange(12, 30))
    else:
        batch = rng.choice([1000, 2048, 4096, 8192])
        c = dict(kind="train", samples=batch * rng.randrange(48, 65) + rng.randrange(batch), batch=batch,
                 epochs=rng.randrange(6, 11))
    c.pop("name", None)
    return c


# ------------------------------------------------------------------ the inputs

def _generator(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _uniform(g, lo, hi, n):
    return lo + (hi - lo) * torch.rand(n, generator=g, device=DEV, dtype=F64)


def _sphere_pack(lx, ly, lz, g, radius=6, target=0.30):
    """Solid mask (z, y, x) of overlapping spheres with uniform centres, periodic in y and z; the
    x faces stay fluid."""
    d = torch.arange(-radius, radius + 1, device=DEV)
    dz, dy, dx = torch.meshgrid(d, d, d, indexing="ij")
    ball = dx * dx + dy * dy + dz * dz <= radius * radius
    count = max(1, int(-math.log(1 - target) * lx * ly * lz / int(ball.sum())))
    x = _uniform(g, 0, lx, count).long()[:, None] + dx[ball][None]
    y = (_uniform(g, 0, ly, count).long()[:, None] + dy[ball][None]) % ly
    z = (_uniform(g, 0, lz, count).long()[:, None] + dz[ball][None]) % lz
    inside = (x >= 1) & (x < lx - 1)
    solid = torch.zeros(lx * ly * lz, dtype=torch.bool, device=DEV)
    solid[(x + lx * (y + ly * z))[inside]] = True
    return solid


def _circles(sizes, fractions, g, tau, rmin=3.0, rmax=12.0):
    """Noble-Torczynski weights of random circles in periodic domains of `sizes` (lx, ly), one after
    the other in one array: cell coverage clamp(r - distance + 1/2, 0, 1), union by maximum."""
    area = math.pi * (rmin * rmin + rmin * rmax + rmax * rmax) / 3
    counts = [max(1, int(-math.log(1 - p) * lx * ly / area)) for (lx, ly), p in zip(sizes, fractions)]
    which = torch.repeat_interleave(torch.arange(len(sizes), device=DEV), torch.tensor(counts, device=DEV))
    lx = torch.tensor([s[0] for s in sizes], device=DEV)[which]
    ly = torch.tensor([s[1] for s in sizes], device=DEV)[which]
    first = torch.tensor(np.concatenate([[0], np.cumsum([a * b for a, b in sizes])])[:-1], device=DEV)[which]
    r = _uniform(g, rmin, rmax, len(which))
    cx, cy = _uniform(g, 0, 1, len(which)) * lx, _uniform(g, 0, 1, len(which)) * ly
    d = torch.arange(-14, 15, device=DEV)
    dy, dx = (a.reshape(1, -1) for a in torch.meshgrid(d, d, indexing="ij"))
    x, y = cx.floor().long()[:, None] + dx, cy.floor().long()[:, None] + dy
    gap = ((x + 0.5 - cx[:, None]) ** 2 + (y + 0.5 - cy[:, None]) ** 2).sqrt()
    cover = (r[:, None] - gap + 0.5).clamp(0, 1)
    at = first[:, None] + x % lx[:, None] + lx[:, None] * (y % ly[:, None])
    eps = torch.zeros(sum(a * b for a, b in sizes), dtype=F64, device=DEV)
    eps.scatter_reduce_(0, at.reshape(-1), cover.reshape(-1), "amax")
    return eps * (tau - 0.5) / ((1 - eps) + (tau - 0.5))


def _solenoidal(side, g, kmax, rms):
    """Random solenoidal field (3, N) from Fourier modes |k| <= kmax, of the given rms."""
    c = torch.arange(side, device=DEV, dtype=F64) * (2 * math.pi / side)
    z, y, x = torch.meshgrid(c, c, c, indexing="ij")
    v = torch.zeros((3, side, side, side), dtype=F64, device=DEV)
    for kx in range(-kmax, kmax + 1):
        for ky in range(-kmax, kmax + 1):
            for kz in range(0, kmax + 1):
                k = torch.tensor([kx, ky, kz], dtype=F64, device=DEV)
                kk = kx * kx + ky * ky + kz * kz
                if kk == 0 or kk > kmax * kmax or (kz == 0 and (ky < 0 or (ky == 0 and kx < 0))):
                    continue
                a = torch.randn(3, generator=g, device=DEV, dtype=F64)
                a = a - k * (a @ k) / kk
                ph = _uniform(g, 0, 2 * math.pi, 1)
                v += a[:, None, None, None] * torch.cos(kx * x + ky * y + kz * z + ph)
    v *= rms / v.square().mean().sqrt()
    return v.reshape(3, -1)


def _network(seed):
    """Parameters of the closure network in the library's layout (W1[32x6], b1, W2[32x32], b2, W3,
    b3): seeded hidden layers, an output near 1."""
    r = np.random.default_rng(seed)
    p = np.zeros(lbmc.MLP_PARAMS, np.float32)
    p[:192] = r.uniform(-0.4, 0.4, 192)
    p[192:224] = r.uniform(-0.1, 0.1, 32)
    p[224:1248] = r.uniform(-0.3, 0.3, 1024)
    p[1248:1280] = r.uniform(-0.1, 0.1, 32)
    p[1280:1312] = r.uniform(-0.1, 0.1, 32)
    p[1312] = 1.0
    return torch.from_numpy(p).bfloat16().float().numpy()


NETWORK_STD, NETWORK_RANGE = 10.0, 4.0


def _flow(case, seed):
    """The flow of a ``step`` case as device tensors and numbers."""
    g = _generator(seed)
    lx, ly, lz = case["lx"], case["ly"], case["lz"]
    n = lx * ly * lz
    w = dict(lattice="d2q9" if lz == 1 else "d3q15", length=(lx, ly, lz), n=n, tau=1.0, tau_mrt=(), c_smag=0.0,
             collision=lbmc.BGK, geometry=None, force=None, macro=None, micro=None, rho=None, u=None, init="rest")
    if case["flow"] == "channel":
        y = torch.arange(n, device=DEV) // lx
        w.update(tau=CHANNEL_TAU, geometry=((y == 0) | (y == ly - 1)).double(),
                 force=torch.zeros((2, n), dtype=F64, device=DEV))
        # the pressure gradient differs from run to run
        w["force"][0] = CHANNEL_G * float(_uniform(g, 0.5, 2.0, 1))
    elif case["flow"] == "porous":
        x = torch.arange(n, device=DEV) % lx
        inlet, outlet = x == 0, x == lx - 1
        w.update(tau=POROUS_TAU, tau_mrt=POROUS_RATES, collision=lbmc.MRT,
                 geometry=_sphere_pack(lx, ly, lz, g).double(),
                 macro=torch.where(inlet | outlet, 8, 0).int(), micro=(inlet.int() + 2 * outlet.int()),
                 rho=1 + (RHO_IN - 1) * inlet.double() + (RHO_OUT - 1) * outlet.double())
    elif case["flow"] == "vortex":
        nu = VORTEX_U0 * lx / (2 * math.pi) / VORTEX_RE
        c = (torch.arange(lx, device=DEV, dtype=F64) + float(_uniform(g, 0, 1, 1))) * (2 * math.pi / lx)
        z, y, x = torch.meshgrid(c, c, c, indexing="ij")
        u = torch.stack([VORTEX_U0 * x.sin() * y.cos() * z.cos(), -VORTEX_U0 * x.cos() * y.sin() * z.cos(),
                         torch.zeros_like(x)])
        p = VORTEX_U0 ** 2 / 16 * ((2 * x).cos() + (2 * y).cos()) * ((2 * z).cos() + 2)
        w.update(tau=0.5 + 3 * nu, c_smag=C_SMAG, init="flow", u=u.reshape(3, n), rho=1 + 3 * p.reshape(n))
    elif case["flow"] == "box":
        w.update(tau=BOX_TAU, c_smag=C_SMAG, init="flow", u=_solenoidal(lx, g, 3, BOX_URMS),
                 rho=torch.ones(n, dtype=F64, device=DEV), force=_solenoidal(lx, g, 2, BOX_AMP),
                 network=_network(seed))
    else:  # obstacles
        w.update(tau=SWEEP_TAU, collision=lbmc.NTPOR, force=torch.zeros((2, n), dtype=F64, device=DEV),
                 geometry=_circles([(lx, ly)], [float(_uniform(g, 0.2, 0.5, 1))], g, SWEEP_TAU))
        w["force"][0] = SWEEP_G
    return w


def _sweep_sizes(case):
    """Side lengths of a ``sweep`` case, log-uniform in [32, 512] per axis (the same for every seed)."""
    r = np.random.default_rng(case["domains"])
    sides = np.rint(np.exp(r.uniform(np.log(32), np.log(512), (case["domains"], 2)))).astype(int)
    return [(int(a), int(b)) for a, b in sides]


def _sweep(case, seed):
    """Sizes and porosities (one flat device array) of a ``sweep`` case."""
    sizes = _sweep_sizes(case)
    fractions = np.random.default_rng(seed).uniform(0.2, 0.5, len(sizes)).tolist()
    return sizes, _circles(sizes, fractions, _generator(seed), SWEEP_TAU)


def _samples(case, seed):
    """Features and targets of a ``train`` case: invariants of random strain-like tensors and an
    eddy viscosity that grows with the strain, with scatter, as the study's samples have it."""
    g = _generator(seed)
    n = case["samples"]
    size = torch.exp(torch.randn(n, generator=g, device=DEV) * 0.8 - 6.5)
    t = torch.randn((n, 6), generator=g, device=DEV) * size[:, None]
    ss = (t[:, :3] ** 2).sum(1) + 2 * (t[:, 3:] ** 2).sum(1)
    x = torch.stack([0.5 * torch.log(2 * ss), torch.log(t.abs().sum(1)), t[:, 0] * t[:, 1] / ss,
                     t[:, :3].sum(1) * 1e3, 0.5 * torch.log((t[:, :3] ** 2).sum(1) + 1e-24),
                     torch.randn(n, generator=g, device=DEV)], 1)
    y = 0.02 * ss.sqrt() * torch.exp(0.3 * torch.randn(n, generator=g, device=DEV))
    return x.cpu().numpy(), y.cpu().numpy(), x.mean(0).cpu().numpy(), x.std(0).cpu().numpy(), float(y.std())


def _host(t):
    """A device tensor in page-locked host memory, as an array."""
    if t is None:
        return None
    out = torch.empty(t.shape, dtype=t.dtype, pin_memory=True)
    out.copy_(t)
    return out.numpy()


def prepare(case, seed):
    if case["kind"] == "step":
        w = _flow(case, seed)
        cfg = lbmc.make_config(w["lattice"], w["length"], tau=w["tau"], tau_mrt=w["tau_mrt"], c_smag=w["c_smag"],
                               collision_type=w["collision"], forcing=w["force"] is not None,
                               macro_bc=w["macro"] is not None, micro_bc=w["micro"] is not None,
                               init_type=lbmc.INIT_EQUILIBRIUM if w["init"] == "flow" else lbmc.INIT_STATIC,
                               storage=case["storage"],
                               streaming=lbmc.STREAM_AA if case["streaming"] == "aa" else lbmc.STREAM_SHIFT)
        dim, q = (2, 9) if w["lattice"] == "d2q9" else (3, 15)
        dom, keep = lbmc.make_domain(w["n"], dim, q, _host(w["geometry"]), _host(w["force"]), _host(w["macro"]),
                                     _host(w["micro"]), _host(w["u"]), _host(w["rho"]))
        engine = lbmc.Engine(cfg, dom)
        del keep
        state = dict(case=case, engine=engine,
                     rho=torch.empty(w["n"], dtype=F64, pin_memory=True).numpy(),
                     u=torch.empty((dim, w["n"]), dtype=F64, pin_memory=True).numpy())
        if case["passes"]:
            m = lbmc.Mlp(seed=1)
            m.set_params(w["network"])
            r = np.full(6, NETWORK_RANGE)
            m.set_normalization(np.zeros(6), np.full(6, NETWORK_STD), -r, r, target_scale=BOX_NU_T)
            m.attach(engine, iterations=case["passes"])
            state["mlp"] = m
        return state
    if case["kind"] == "sweep":
        sizes, B = _sweep(case, seed)
        B = B.cpu().numpy()
        geoms, at = [], 0
        for lx, ly in sizes:
            geoms.append(B[at:at + lx * ly].reshape(ly, lx))
            at += lx * ly
        return dict(case=case, geoms=geoms)
    x, y, mean, std, scale = _samples(case, seed)
    m = lbmc.Mlp(seed=1)
    m.set_normalization(mean, std, target_scale=scale)
    return dict(case=case, mlp=m, x=x, y=y, start=_network(seed))


def run(state):
    case = state["case"]
    if case["kind"] == "step":
        e = state["engine"]
        e.iterate(case["steps"], lbmc.STORE_MACROS | lbmc.REDUCE_DIAG | lbmc.SYNC)
        d = e.diag()
        rho, u = torch.from_numpy(e.rho(out=state["rho"])), torch.from_numpy(e.u(out=state["u"]))
        kind = F64 if case["storage"] == "f64" else torch.float32
        return dict(rho=rho.to(kind), u=u.to(kind), sums=torch.tensor([d.mass, d.kinetic_energy]).to(kind))
    if case["kind"] == "sweep":
        with lbmc.Batch(state["geoms"], tau=SWEEP_TAU, force=(SWEEP_G, 0.0), storage=case["storage"]) as b:
            res = b.run(case["cap"], SWEEP_TOL, SWEEP_CHECK)
            ux = np.concatenate([b.fetch(d, lbmc.FIELD_U_X) for d in range(b.n)])
        return dict(ux=torch.from_numpy(ux).float(), steps=np.array([r.steps for r in res]),
                    delta_u=np.array([r.delta_u for r in res], np.float32))
    m = state["mlp"]
    m.set_params(state["start"])
    grads, loss = m.gradients(state["x"], state["y"])
    history = m.train(state["x"], state["y"], epochs=case["epochs"], batch=case["batch"], lr=TRAIN_LR)
    return dict(grads=grads, loss=np.float32(loss), history=history, params=m.params())


# Operations of one node update in each flow (multiplies and additions of the collision, counted
# from the formulas: moments, equilibria, relaxation, source terms).
FLOPS = dict(channel=190, porous=300, vortex=430, box=430, obstacles=230, sweep=230)
NETWORK_FLOPS = 2 * (6 * 32 + 32 * 32 + 32) + 100


def work(case):
    """The state is read once and written once in a pass (a call of many steps needs no more of the
    memory), the fields come out once; every step updates every node."""
    size = {"f64": 8, "f32": 4}.get(case.get("storage"), 2)
    if case["kind"] == "step":
        n = case["lx"] * case["ly"] * case["lz"]
        q, dim = (9, 2) if case["lz"] == 1 else (15, 3)
        out = 8 if case["storage"] == "f64" else 4
        return {"bytes": n * (2 * q * size + 1 + out * (dim + 1)),
                "flops": n * case["steps"] * (FLOPS[case["flow"]] + case["passes"] * NETWORK_FLOPS)}
    if case["kind"] == "sweep":
        n = sum(a * b for a, b in _sweep_sizes(case))
        return {"bytes": n * (2 * 9 * size + 8 + 4), "flops": n * case["cap"] * FLOPS["sweep"]}
    n, batches = case["samples"], case["samples"] // case["batch"] * case["epochs"]
    # forward, and backward through both layers, for the gradient and for each epoch
    return {"bytes": n * 28 * (1 + case["epochs"]) + 1313 * 16 * batches,
            "flops": 3 * NETWORK_FLOPS * (n + batches * case["batch"])}


# ------------------------------------------------------- the same in 64 bits

E2 = [(0, 0), (1, 0), (0, 1), (-1, 0), (0, -1), (1, 1), (-1, 1), (-1, -1), (1, -1)]
E3 = [(0, 0, 0), (1, 0, 0), (-1, 0, 0), (0, 1, 0), (0, -1, 0), (0, 0, 1), (0, 0, -1), (1, 1, 1), (-1, 1, 1),
      (1, -1, 1), (-1, -1, 1), (1, 1, -1), (-1, 1, -1), (1, -1, -1), (-1, -1, -1)]
# Signs of the tangential terms of the x pressure faces, as LBM-C/boundary_conditions/d3q15 has them.
FACE_SIGNS = {1: {7: (-1, 1), 11: (-1, -1), 9: (1, 1), 13: (1, -1)},
              -1: {14: (1, -1), 10: (1, 1), 12: (-1, 1), 8: (-1, -1)}}


class _Exact:
    """The lattice Boltzmann step on deviations g = f - w in 64 bits, one time step per call.

    ``move``: streams the populations (one periodic box, or several boxes one after the other)."""

    def __init__(self, dim, n, tau, move, rates=None, c_smag=0.0, solid=None, B=None, force=None, faces=None,
                 closure=None):
        self.e = torch.tensor(E2 if dim == 2 else E3, dtype=F64, device=DEV)
        norm = self.e.abs().sum(1)
        self.w = (torch.where(norm == 0, 16.0, torch.where(norm == 1, 4.0, 1.0)).double() / 36 if dim == 2 else
                  torch.where(norm == 0, 16.0, torch.where(norm == 1, 8.0, 1.0)).double() / 72)
        el = self.e.long().tolist()
        self.opp = [el.index([-v for v in c]) for c in el]
        self.dim, self.q, self.n, self.tau, self.move = dim, len(el), n, tau, move
        self.c_smag, self.solid, self.B, self.force, self.faces, self.closure = c_smag, solid, B, force, faces, closure
        if rates is not None:
            self.rates = torch.tensor(rates, dtype=F64, device=DEV)
            self.m = self._moments15()
        else:
            self.rates = None

    def _moments15(self):
        x, y, z = self.e.T
        c2 = self.e.square().sum(1)
        flux = torch.where(c2 == 1, -4.0, 1.0).double()
        return torch.stack([torch.ones_like(x), torch.where(c2 == 0, -2.0, torch.where(c2 == 1, -1.0, 1.0)).double(),
                            torch.where(c2 == 0, 16.0, torch.where(c2 == 1, -4.0, 1.0).double()), x, x * flux, y, y * flux, z,
                            z * flux, 3 * x * x - c2, y * y - z * z, x * y, y * z, x * z, x * y * z])

    def equilibrium(self, drho, u):
        """g_eq for each population, (q, n)."""
        eu = 3 * (self.e @ u)
        usq = 1.5 * u.square().sum(0)
        rho = 1 + drho
        return self.w[:, None] * (drho + rho * (eu + 0.5 * eu * eu - usq))

    def pressure_face(self, g, at, rho, sign):
        """Zou-He pressure face normal to x (sign +1: low face) at the nodes `at`."""
        f = g[:, at]
        drho = rho - 1
        i0, i1 = (1, 2) if sign > 0 else (2, 1)  # inward, outward along x
        out = [k for k in range(15) if self.e[k, 0] == -sign]
        flat = [k for k in range(15) if self.e[k, 0] == 0]
        ux = sign * (drho - f[flat].sum(0) - 2 * f[out].sum(0)) / rho
        ru = rho * ux
        a, b = f[3] - f[4], f[5] - f[6]
        f[i0] = f[i1] + sign * 2 / 3 * ru
        for k, (ca, cb) in FACE_SIGNS[sign].items():
            f[k] = f[self.opp[k]] + sign * ru / 12 - 0.25 * (ca * a + cb * b)
        g[:, at] = f
        return ux

    def step(self, g, streamed):
        if streamed:
            g = self.move(g)
        drho = g.sum(0)
        u = (self.e.T @ g) / (1 + drho)
        for at, rho, sign in self.faces or []:
            drho[at] = rho - 1
            u[:, at] = 0
            u[0, at] = self.pressure_face(g, at, rho, sign)
        rho = 1 + drho
        source = None
        if self.force is not None:
            F = self.force
            u = u + F / (2 * rho)
            eF, eu, uF = self.e @ F, self.e @ u, (u * F).sum(0)
            pre = 1 - 1 / (2 * self.tau)
            source = self.w[:, None] * pre * (3 * (eF - uF) + 9 * eu * eF)
        if self.rates is not None:
            j = rho * u
            jj = j.square().sum(0)
            c = -7.0 / 3.0
            meq = torch.stack([drho, -drho + jj, drho - 5 * jj, j[0], c * j[0], j[1], c * j[1], j[2], c * j[2],
                               3 * j[0] * j[0] - jj, j[1] * j[1] - j[2] * j[2], j[0] * j[1], j[1] * j[2], j[0] * j[2],
                               torch.zeros_like(jj)])
            change = (self.m.T * (self.rates / self.m.square().sum(1))) @ (self.m @ g - meq)
        else:
            neq = g - self.equilibrium(drho, u)
            tau = self.tau
            if self.c_smag > 0:
                pairs = [(0, 0), (1, 1), (2, 2), (0, 1), (1, 2), (0, 2)]
                s = torch.stack([self.e[:, a] * self.e[:, b] for a, b in pairs]) @ neq
                weight = torch.tensor([1, 1, 1, 2, 2, 2], dtype=F64, device=DEV)
                root2 = math.sqrt(2.0)
                strain = root2 * (weight @ s.abs())
                tau = self.tau + 0.5 * ((self.tau ** 2 + 18 * root2 * self.c_smag ** 2 * strain / rho).sqrt() - self.tau)
                if self.closure is not None:
                    tau = self.closure(s, rho, tau, self.tau)
            change = neq / tau
        if self.B is None:
            new = g - change
            if source is not None:
                new += source
        else:
            new = g - (1 - self.B) * (change - source) + self.B * (g[self.opp] - g)
        if self.solid is not None:
            new = torch.where(self.solid, g[self.opp], new)
            rho = torch.where(self.solid, 0.0, rho)
            u = torch.where(self.solid, 0.0, u)
        return new, rho, u


def _closure(params, passes):
    p = torch.from_numpy(params).to(DEV).double()
    w1, b1, w2, b2, w3, b3 = p[:192].reshape(32, 6), p[192:224], p[224:1248].reshape(32, 32), p[1248:1280], p[1280:1312], p[1312]

    def tau_of(s, rho, tau_smag, tau0):
        tau, inside = tau_smag, torch.ones_like(rho, dtype=torch.bool)
        for _ in range(passes):
            xx, yy, zz, xy, yz, xz = -1.5 / (rho * tau) * s
            d2 = xx * xx + yy * yy + zz * zz
            ss = d2 + 2 * (xy * xy + yz * yz + xz * xz)
            total = xx.abs() + yy.abs() + zz.abs() + 2 * (xy.abs() + yz.abs() + xz.abs())
            det = xx * (yy * zz - yz * yz) - xy * (xy * zz - yz * xz) + xz * (xy * yz - yy * xz)
            x = torch.stack([0.5 * torch.log(2 * ss + 1e-24), torch.log(1e-12 + total),
                             torch.copysign(torch.log(1 + det.abs() * 1e9), det), (xx + yy + zz) * 1e3,
                             0.5 * torch.log(d2 + 1e-24), (rho - 1) * 1e2]) / NETWORK_STD
            inside = inside & (x.abs() <= NETWORK_RANGE).all(0)
            silu = torch.nn.functional.silu
            y = w3 @ silu(w2 @ silu(w1 @ x + b1[:, None]) + b2[:, None]) + b3
            tau = torch.where(inside, tau0 + 3 * (BOX_NU_T * y).clamp(min=0), tau)
        return torch.where(inside, tau, tau_smag)

    return tau_of


def _exact_step(case, seed):
    w = _flow(case, seed)
    dim = 2 if w["lattice"] == "d2q9" else 3
    shape = tuple(reversed(w["length"][:dim]))  # (z,) y, x
    e = E2 if dim == 2 else E3

    def move(g):
        axes = tuple(range(dim))
        return torch.stack([torch.roll(g[i].reshape(shape), tuple(reversed(c)), axes).reshape(-1) for i, c in enumerate(e)])

    solid = B = faces = None
    if w["geometry"] is not None:
        solid = w["geometry"] >= 1
        if w["collision"] == lbmc.NTPOR:
            B = w["geometry"]
    if w["micro"] is not None:
        faces = [(torch.nonzero(w["micro"] == 1)[:, 0], RHO_IN, 1), (torch.nonzero(w["micro"] == 2)[:, 0], RHO_OUT, -1)]
    rates = w["tau_mrt"] if w["collision"] == lbmc.MRT else None
    x = _Exact(dim, w["n"], w["tau"], move, rates, w["c_smag"], solid, B, w["force"], faces,
               _closure(w["network"], case["passes"]) if case["passes"] else None)
    g = (x.equilibrium(w["rho"] - 1, w["u"]) if w["init"] == "flow" else
         torch.zeros((x.q, w["n"]), dtype=F64, device=DEV))
    for t in range(case["steps"]):
        g, rho, u = x.step(g, t > 0)
    sums = torch.stack([rho.sum(), 0.5 * (rho * u.square().sum(0)).sum()])
    return dict(rho=rho, u=u, sums=sums)


def _exact_sweep(case, seed):
    sizes, B = _sweep(case, seed)
    n = len(B)
    which = torch.repeat_interleave(torch.arange(len(sizes), device=DEV),
                                    torch.tensor([a * b for a, b in sizes], device=DEV))
    lx, ly = (torch.tensor([s[k] for s in sizes], device=DEV)[which] for k in (0, 1))
    first = torch.tensor(np.concatenate([[0], np.cumsum([a * b for a, b in sizes])])[:-1], device=DEV)[which]
    k = torch.arange(n, device=DEV) - first
    x, y = k % lx, k // lx
    source = [first + (x - c[0]) % lx + lx * ((y - c[1]) % ly) for c in E2]
    force = torch.zeros((2, 1), dtype=F64, device=DEV)
    force[0] = SWEEP_G
    s = _Exact(2, n, SWEEP_TAU, lambda g: torch.stack([g[i][at] for i, at in enumerate(source)]), None, 0.0, B >= 1, B,
               force)
    g = torch.zeros((9, n), dtype=F64, device=DEV)
    kept, frozen = None, torch.zeros(len(sizes), dtype=torch.bool, device=DEV)
    for t in range(case["cap"]):
        new, _, u = s.step(g, t > 0)
        # a domain that converged stays as it was after the step that showed it
        g = torch.where(frozen[which], g, new)
        if t % SWEEP_CHECK == 0:
            if kept is not None:
                worst = torch.zeros(len(sizes), dtype=F64, device=DEV)
                worst.scatter_reduce_(0, which, (u - kept).abs().amax(0), "amax")
                frozen |= worst < SWEEP_TOL
            kept = u
    g = s.move(g)
    return dict(ux=(s.e[:, 0] @ g) / (1 + g.sum(0)), steps=None, delta_u=None)


def _exact_train(case, seed):
    x, y, mean, std, scale = _samples(case, seed)
    p = torch.from_numpy(_network(seed)).to(DEV).double().requires_grad_(True)
    w1, b1, w2, b2, w3, b3 = p[:192].reshape(32, 6), p[192:224], p[224:1248].reshape(32, 32), p[1248:1280], p[1280:1312], p[1312]
    xn = (torch.from_numpy(x).to(DEV).double() - torch.from_numpy(mean).to(DEV).double()) / torch.from_numpy(std).to(DEV).double()
    t = torch.from_numpy(y).to(DEV).double() / scale
    silu = torch.nn.functional.silu
    out = silu(silu(xn @ w1.T + b1) @ w2.T + b2) @ w3 + b3
    loss = (out - t).square().mean()
    loss.backward()
    return dict(grads=p.grad, loss=loss.detach(), history=None, params=None)


def exact(case, seed):
    if case["kind"] == "step":
        return _exact_step(case, seed)
    if case["kind"] == "sweep":
        return _exact_sweep(case, seed)
    return _exact_train(case, seed)
