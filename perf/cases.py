"""Measured cases of the sampler: what programs built on libclbm do, through
its public entry points (the clbm package, ctypes over the C ABI).

Kinds of pass:
  step     one LB step of a program that calls the reference's functions one by
           one on a single state (device arrays): collide and stream, walls,
           square, interior, drag
  perturb  one generatePerturbedState call on a device state
  warmup   the warm-up / snapshot generator: one state loaded, stepped, its
           macroscopic fields and the state read back
  driver   one cloning interval as the drop-in drivers run it: interval, drag
           series, cloning step, copy numbers, slot 0's new state
  batch    one cloning interval of a large population, every output delivered
           (clbm_run_sampler_outputs), captured as a CUDA graph; slot 0's new
           state
  adjoint  the drag integral forward and backward, every clone's gradient

Initial states are the repository's synthetic ones: equilibrium at rho = 1,
u = (u0, 0) with a relative noise per population.  A context is tuned once
(clbm_autotune) when it is made, as the drivers and the benchmark do.
"""
from __future__ import annotations

import math
import random
import sys
from pathlib import Path

import numpy as np
import torch

_PKG = str(Path(__file__).resolve().parent.parent / "cloning-lbm-mpi_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)
import clbm  # noqa: E402
from clbm.configs import Run  # noqa: E402

NOISE = 1e-3  # of the initial states


def listed():
    return [
        # the reference's square lattice for L = 32, one LB step through its own functions: the smallest call
        dict(name="step_129x129", kind="step", width=129, height=129, side=32, tau=0.56),
        # generatePerturbedState on a 257 x 257 state, ten snapshots as the population-perturbation driver keeps
        dict(name="perturb_257x257", kind="perturb", width=257, height=257, nsnap=10),
        # the warm-up generator writing one snapshot: a single FP64 state, where little of the GPU has work
        dict(name="warmup_129x129_fp64", kind="warmup", width=129, height=129, side=32, tau=0.56, steps=100, fp32=False),
        # the plain FP64 cloning run of the repository's configurations: a few clones
        dict(name="driver_16x200x50_fp64", kind="driver", lattices="200x50", side=8, clones=16, ranks=1, tau=0.56,
             k=0.1, steps=100, fp32=False, mix=False, systematic=False, momentum=False),
        # the population-perturbation driver: odd square lattice, four virtual ranks, snapshot mix
        dict(name="driver_32x101x101_mix", kind="driver", lattices="101x101", side=25, clones=32, ranks=4, tau=0.55,
             k=0.1, steps=40, fp32=False, mix=True, systematic=False, momentum=False),
        # the FP64 mode on an ordinary population (the reference's arithmetic, bit for bit)
        dict(name="driver_256x256x64_fp64", kind="driver", lattices="256x64", side=12, clones=256, ranks=1, tau=0.55,
             k=0.3, steps=50, fp32=False, mix=False, systematic=False, momentum=False),
        # a small FP32 run, odd channel, momentum-exchange drag and systematic resampling
        dict(name="driver_64x97x33_fp32", kind="driver", lattices="97x33", side=6, clones=64, ranks=1, tau=0.56,
             k=0.5, steps=50, fp32=True, mix=False, systematic=True, momentum=True),
        # the headline: 4096 clones of 256 x 64
        dict(name="batch_4096x256x64", kind="batch", lattices="256x64", side=12, clones=4096, runs=1, tau=0.55,
             k=0.3, steps=100, field_steps=0),
        # two biases on the shedding 400 x 100 channel, long intervals
        dict(name="batch_2x512x400x100", kind="batch", lattices="400x100", side=20, clones=512, runs=2, tau=0.53,
             k=0.2, steps=200, field_steps=0),
        # eight uneven lattices in one context
        dict(name="batch_uneven_8x256", kind="batch",
             lattices="128x32,192x48,256x64,320x80,384x96,448x112,512x128,256x128", side=0, clones=256, runs=1,
             tau=0.55, k=0.5, steps=100, field_steps=0),
        # the forcing variant: a random body-force field per clone and interval
        dict(name="batch_4096x256x64_field", kind="batch", lattices="256x64", side=12, clones=4096, runs=1, tau=0.55,
             k=0.3, steps=100, field_steps=20),
        # gradient of the drag integral with respect to the initial populations
        dict(name="adjoint_64x400x100", kind="adjoint", width=400, height=100, side=20, clones=64, tau=0.56,
             steps=200, every=20, fp32=True),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def _lattice(rng, lo_w, hi_w, lo_h, hi_h):
    w, h = _log_int(rng, lo_w, hi_w), _log_int(rng, lo_h, hi_h)
    return w, h, max(3, min(w // 3, h // 5 + rng.randint(-1, 1)))


def draw(rng: random.Random) -> dict:
    kind = rng.choice(["step", "perturb", "warmup", "driver", "driver", "driver", "batch", "batch", "batch", "adjoint"])
    tau = rng.choice([0.53, 0.55, 0.56, 0.6])
    if kind in ("step", "warmup"):
        w, h, side = _lattice(rng, 48, 400, 24, 300)
        c = dict(kind=kind, width=w, height=h, side=side, tau=tau)
        return c if kind == "step" else dict(c, steps=rng.randint(20, 200), fp32=rng.random() < 0.3)
    if kind == "perturb":
        w, h, _ = _lattice(rng, 48, 400, 24, 300)
        return dict(kind=kind, width=w, height=h, nsnap=rng.randint(2, 16))
    if kind == "driver":
        w, h, side = _lattice(rng, 48, 300, 24, 128)
        fp32 = rng.random() < 0.4
        most = (8_000_000 if fp32 else 4_200_000) // (w * h)
        ranks = rng.choice([1, 1, 2, 4])
        mix = rng.random() < 0.4
        return dict(kind=kind, lattices=f"{w}x{h}", side=side, clones=ranks * max(1, _log_int(rng, 8, max(9, most)) // ranks),
                    ranks=ranks, tau=tau, k=rng.choice([-0.2, 0.1, 0.3, 0.5]), steps=rng.randint(20, 60), fp32=fp32,
                    mix=mix, systematic=rng.random() < 0.4, momentum=rng.random() < 0.3)
    if kind == "batch":
        n = rng.choice([1, 1, 2, 5])
        lats = [_lattice(rng, 96, 512, 32, 128) for _ in range(n)]
        nodes = sum(w * h for w, h, _ in lats)
        return dict(kind=kind, lattices=",".join(f"{w}x{h}" for w, h, _ in lats), side=0,
                    clones=_log_int(rng, 48, min(4096, 50_000_000 // nodes)), runs=1, tau=tau,
                    k=rng.choice([-0.5, 0.2, 0.3]), steps=rng.randint(40, 100),
                    field_steps=rng.choice([0, 0, 0, 15]))
    w, h, side = _lattice(rng, 96, 400, 40, 100)
    fp32 = rng.random() < 0.7
    return dict(kind="adjoint", width=w, height=h, side=side, clones=_log_int(rng, 4, 64 if fp32 else 16), tau=tau,
                steps=rng.randint(20, 150), every=rng.randint(7, 30), fp32=fp32)


# ---------------------------------------------------------------- inputs ----
def _u0(c):
    return 0.04 if c["tau"] == 0.55 else 0.05


def _runs(c, seed):
    """The clbm.configs runs of a sampler case."""
    lats = [tuple(map(int, s.split("x"))) for s in c["lattices"].split(",")]
    many = len(lats) * c.get("runs", 1)
    out = []
    for i in range(many):
        w, h = lats[i % len(lats)]
        k = c["k"] if many == 1 else c["k"] * (2.0 * i / (many - 1) - 1.0)  # evenly over [-k, k]
        out.append(Run(w, h, c["side"] or h // 5, w // 4, h // 2, c["clones"], _u0(c), c["tau"], k, 1e-5, seed % 100003 + 1,
                       perturb_mode=clbm.PERTURB_MIX if c.get("mix") else clbm.PERTURB_UNIFORM,
                       resample_mode=clbm.RESAMPLE_SYSTEMATIC if c.get("systematic") else clbm.RESAMPLE_REFERENCE,
                       field_steps=c.get("field_steps", 0), field_eps=0.1, field_sigma=32.0))
    return out


def _descs(c, seed):
    out = []
    for r in _runs(c, seed):
        d = r.desc()
        d.ranks = c.get("ranks", 1)
        d.drag_mode = clbm.DRAG_MOMENTUM if c.get("momentum") else clbm.DRAG_STRESS
        d.nsnap = 10 if c.get("mix") else 0
        d.eps = 1e-3 if c.get("mix") else d.eps
        out.append(d)
    return out


def _geometry(c):
    """width, height and the square's xmin, xmax, ymin, ymax (perimeter inclusive) of a single-state case."""
    w, h, s = c["width"], c["height"], c["side"]
    return w, h, w // 4 - s // 2, w // 4 - s // 2 + s, h // 2 - s // 2, h // 2 - s // 2 + s


def _single(c, seed):
    """One run over a single lattice (warmup, adjoint)."""
    r = Run(c["width"], c["height"], c["side"], c["width"] // 4, c["height"] // 2, c.get("clones", 1), _u0(c), c["tau"], 0.0,
            0.0, seed % 100003 + 1, perturb_mode=clbm.PERTURB_NONE)
    return r.desc(), r


def _states(w, h, n, seed):
    """n noisy states at rest with a developed mean flow, [n][w][h][9] FP64 on the GPU."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    y = torch.linspace(0.0, math.pi, h, dtype=torch.float64, device="cuda")
    u = 0.06 * torch.sin(y)[None, None, :].expand(n, w, h)
    f = torch.stack(_equilibrium(torch.ones_like(u), u, torch.zeros_like(u)), dim=-1)
    return f * (1.0 + NOISE * (2.0 * torch.rand(f.shape, dtype=torch.float64, device="cuda", generator=g) - 1.0))


def prepare(case, seed):
    c, kind = case, case["kind"]
    if kind == "step":
        w, h, *box = _geometry(c)
        f = _states(w, h, 1, seed)[0].contiguous()
        macro = torch.empty(3, w * h, dtype=torch.float64, device="cuda")
        return dict(kind=kind, g=clbm.geom(w, h, *box), f=f, g2=torch.empty_like(f), macro=macro, tau=c["tau"], beta=1e-6)
    if kind == "perturb":
        w, h, n = c["width"], c["height"], c["nsnap"]
        s = _states(w, h, n + 1, seed)
        return dict(kind=kind, f=s[0].contiguous(), snaps=s[1:].contiguous(), n=n, size=9 * w * h,
                    pre=np.random.default_rng(seed).random(n))
    if kind == "warmup":
        d, _ = _single(c, seed)
        s = clbm.Sampler([d], clbm.FP32 if c["fp32"] else clbm.FP64, max_steps=c["steps"])
        s.autotune(launches=3, measure=False)
        return dict(kind=kind, s=s, f=_states(c["width"], c["height"], 1, seed).cpu().numpy().reshape(-1), steps=c["steps"])
    if kind == "adjoint":
        d, r = _single(c, seed)
        s = clbm.Sampler([d], clbm.FP32 if c["fp32"] else clbm.FP64, max_steps=c["steps"])
        s.init_equilibrium(0, r.u0, NOISE, seed)
        s.autotune(launches=3, measure=False)
        return dict(kind=kind, s=s, steps=c["steps"], every=c["every"], clones=c["clones"])
    runs, descs = _runs(c, seed), _descs(c, seed)
    fp32 = c.get("fp32", True)
    s = clbm.Sampler(descs, clbm.FP32 if fp32 else clbm.FP64, max_steps=c["steps"],
                     flags=clbm.FLAG_GRAPH if kind == "batch" else 0)
    for i, r in enumerate(runs):
        s.init_equilibrium(i, r.u0, NOISE, seed)
        if c.get("mix"):
            s.set_snapshots(i, _states(r.width, r.height, 10, seed + i).cpu().numpy())
    s.autotune(launches=3, measure=False)
    return dict(kind=kind, s=s, steps=c["steps"], runs=len(runs), out={})


def run(state):
    t, kind = state, state["kind"]
    if kind == "step":
        g, f, f2, m = t["g"], t["f"], t["g2"], t["macro"]
        clbm.ref_stream_collide(g, f.data_ptr(), f2.data_ptr(), m[0].data_ptr(), m[1].data_ptr(), m[2].data_ptr(),
                                t["beta"], t["tau"])
        clbm.ref_walls_bb(g, f2.data_ptr(), f.data_ptr())
        clbm.ref_square_bb(g, f2.data_ptr(), f.data_ptr())
        clbm.ref_interior_reset(g, f2.data_ptr())
        force = clbm.ref_force_on_square(g, f2.data_ptr(), 1.0 / t["tau"])
        t["f"], t["g2"] = f2, f
        return dict(post=f, state=f2, macro=m, force=force)
    if kind == "perturb":
        clbm.ref_perturbed_state(t["f"].data_ptr(), t["snaps"].data_ptr(), 1e-3, t["n"], t["size"], t["pre"])
        return dict(state=t["f"])
    s = t["s"]
    if kind == "warmup":
        s.load(0, 0, t["f"])
        s.run_interval(t["steps"])
        drag = s.drag(0)
        rho, ux, uy = s.macro(0, 0)
        return dict(drag=drag, rho=rho, ux=ux, uy=uy, state=s.dump(0, 0))
    if kind == "adjoint":
        J = s.drag_fwd(t["steps"], t["every"])
        s.drag_bwd()
        return dict(J=J, grad=np.stack([s.drag_grad(0, j) for j in range(t["clones"])]))
    if kind == "driver":
        s.run_interval(t["steps"])
        drag = s.drag(0)
        s.clone_step()
        r = s.clone_result(0)
        return dict(r, drag=drag, state=s.dump(0, 0))
    return dict(s.run_sampler_outputs(t["steps"], 1, t["out"]), state=s.dump(0, 0))


# ------------------------------------------------------------------ work ----
def work(case):
    """Bytes: every state read once and written once, the outputs written once.
    Flops: per node and step the BGK / Guo collision's additions and products
    (about 130), twice that and a recomputed forward for the adjoint."""
    c, kind = case, case["kind"]
    if kind == "step":
        n = c["width"] * c["height"]
        return dict(bytes=n * 8 * (9 + 18 + 3), flops=130.0 * n)
    if kind == "perturb":
        n = 9 * c["width"] * c["height"]
        return dict(bytes=8.0 * n * (c["nsnap"] + 2), flops=(2.0 * c["nsnap"] + 4) * n)
    if kind == "warmup":
        n = c["width"] * c["height"]
        return dict(bytes=8.0 * n * (9 + 9 + 3) + 8 * c["steps"], flops=130.0 * n * c["steps"])
    if kind == "adjoint":
        n = c["width"] * c["height"] * c["clones"]
        e = 4 if c["fp32"] else 8
        return dict(bytes=n * 9.0 * (e + 8), flops=3 * 130.0 * n * c["steps"])
    lats = [tuple(map(int, s.split("x"))) for s in c["lattices"].split(",")]
    n = sum(w * h for w, h in lats) * c["clones"] * c.get("runs", 1)
    clones = len(lats) * c["clones"] * c.get("runs", 1)
    e = 4 if c.get("fp32", True) else 8
    return dict(bytes=n * 18.0 * e + clones * (8.0 * c["steps"] + 20), flops=130.0 * n * c["steps"])


# ----------------------------------------------------------------- exact ----
CX = (0, 1, 0, -1, 0, 1, -1, -1, 1)
CY = (0, 0, 1, 0, -1, 1, 1, -1, -1)
OPP = (0, 3, 4, 1, 2, 7, 8, 5, 6)
WT = (4 / 9,) + (1 / 9,) * 4 + (1 / 36,) * 4


def _equilibrium(rho, ux, uy):
    u2 = 1.5 * (ux * ux + uy * uy)
    out = []
    for k in range(9):
        e = CX[k] * ux + CY[k] * uy
        out.append(WT[k] * rho * (1.0 + 3.0 * e + 4.5 * e * e - u2))
    return out


def _moments(f):
    rho = sum(f)
    return rho, sum(CX[k] * f[k] for k in range(9) if CX[k]), sum(CY[k] * f[k] for k in range(9) if CY[k])


def _masks(h, w, box):
    """[9][h][w] slots that bounce back, and the square's interior."""
    x0, x1, y0, y1 = box
    m = torch.zeros(9, h, w, dtype=torch.bool, device="cuda")
    for k in (4, 7, 8):
        m[k, h - 1, :] = True
        m[k, y0, x0 + 1:x1] = True
    for k in (2, 5, 6):
        m[k, 0, :] = True
        m[k, y1, x0 + 1:x1] = True
    for k in (3, 6, 7):
        m[k, y0 + 1:y1, x0] = True
    for k in (1, 5, 8):
        m[k, y0 + 1:y1, x1] = True
    m[7, y0, x0] = m[6, y1, x0] = m[5, y1, x1] = m[8, y0, x1] = True
    solid = torch.zeros(h, w, dtype=torch.bool, device="cuda")
    solid[y0 + 1:y1, x0 + 1:x1] = True
    return m, solid


def _collide(f, beta, tau):
    om = 1.0 / tau
    rho, jx, jy = _moments(f)
    ux, uy = (jx + 0.5 * beta) / rho, jy / rho
    feq = _equilibrium(rho, ux, uy)
    post = []
    for k in range(9):
        e = CX[k] * ux + CY[k] * uy
        g = WT[k] * (1.0 - 0.5 * om) * beta * (3.0 * (CX[k] - ux) + 9.0 * CX[k] * e)
        post.append((1.0 - om) * f[k] + om * feq[k] + g)
    return post, rho, ux, uy


def _stream(post, masks, solid):
    out = []
    for k in range(9):
        s = torch.roll(post[k], (CY[k], CX[k]), (-2, -1))
        s = torch.where(masks[k], post[OPP[k]], s)
        out.append(torch.where(solid, torch.full_like(s, WT[k]), s))
    return out


def _force(f, box, tau, masks=None):
    """Drag of every state: stress integration, or momentum exchange where masks is given."""
    x0, x1, y0, y1 = box
    if masks is not None:
        ring = [torch.where(masks[k, y0:y1 + 1, x0:x1 + 1], f[k][..., y0:y1 + 1, x0:x1 + 1], 0.0) * (-2.0 * CX[k])
                for k in range(9) if CX[k]]
        return sum(ring).sum((-2, -1))
    c = 1.0 - 0.5 / tau

    def terms(sl):
        g = [v[sl] for v in f]
        rho, jx, jy = _moments(g)
        feq = _equilibrium(rho, jx / rho, jy / rho)
        n = [a - b for a, b in zip(g, feq)]
        return rho, n[1] + n[3] + n[5] + n[6] + n[7] + n[8], n[5] - n[6] + n[7] - n[8]

    rw, xw, _ = terms((..., slice(y0, y1 + 1), x0))
    re, xe, _ = terms((..., slice(y0, y1 + 1), x1))
    _, _, pn = terms((..., y1, slice(x0, x1 + 1)))
    _, _, ps = terms((..., y0, slice(x0, x1 + 1)))
    return (rw / 3 + c * xw).sum(-1) - (re / 3 + c * xe).sum(-1) - c * pn.sum(-1) + c * ps.sum(-1)


def _philox(seed, c0, c1, c2, c3):
    """Philox4x32-10 on int64 tensors holding 32-bit words; the first two words."""
    m = 0xFFFFFFFF
    k0, k1 = seed & m, (seed >> 32) & m
    c = [c0, c1, c2, c3]
    for _ in range(10):
        p0, p1 = c[0] * 0xD2511F53, c[2] * 0xCD9E8D57
        c = [((p1 >> 32) & m) ^ c[1] ^ k0, p1 & m, ((p0 >> 32) & m) ^ c[3] ^ k1, p0 & m]
        k0, k1 = (k0 + 0x9E3779B9) & m, (k1 + 0xBB67AE85) & m
    return c[0], c[1]


def _initial(r, box, run, seed, first, count):
    """States of clones [first, first + count) of a run as clbm_init_equilibrium makes them: nine [count][h][w]."""
    w, h = r.width, r.height
    _, solid = _masks(h, w, box)
    x = torch.arange(w, device="cuda")[None, None, :]
    y = torch.arange(h, device="cuda")[None, :, None]
    clone = torch.arange(first, first + count, device="cuda")[:, None, None]
    out = []
    one = torch.ones((), dtype=torch.float64, device="cuda")
    feq = _equilibrium(one, r.u0 * one, 0.0 * one)
    for k in range(9):
        idx = (k + 9 * (y + h * x)).expand(count, h, w)
        a, b = _philox(seed, idx, clone.expand(count, h, w), torch.full_like(idx, 0xFFFFFFFF),
                       torch.full_like(idx, (run << 4) | 1))
        u = (((a >> 5) << 26) | (b >> 6)).double() * 2.0 ** -53
        out.append(torch.where(solid, torch.full_like(u, WT[k]), feq[k] * (1.0 + NOISE * (2.0 * u - 1.0))))
    return out


def _fields(r, run, seed, first, count):
    """Random fields of interval 0, [count][h][w]: circulant embedding of the Gaussian covariance."""
    w, h = r.width, r.height
    m1, m2 = 2 * w - 1, 2 * h - 1

    def spectrum(m):
        j = torch.arange(m, dtype=torch.float64, device="cuda")
        d = torch.minimum(j, m - j)
        return torch.fft.fft(torch.exp(-d * d / (2 * r.field_sigma ** 2))).real

    lam = (spectrum(m1)[:, None] * spectrum(m2)[None, :] / (m1 * m2)).clamp_min(0.0).sqrt()
    idx = torch.arange(m1 * m2, device="cuda").reshape(1, m1, m2).expand(count, m1, m2)
    clone = torch.arange(first, first + count, device="cuda")[:, None, None].expand(count, m1, m2)
    a, b = _philox(seed, idx, clone, torch.zeros_like(idx), torch.full_like(idx, (run << 4) | 4))
    rad = torch.sqrt(-2.0 * torch.log((a.float() + 1.0).double() * 2.0 ** -32)) * lam
    ang = 2.0 * math.pi * (b.float().double() * 2.0 ** -32)
    z = torch.fft.fft2(torch.complex(rad * torch.cos(ang), rad * torch.sin(ang))).real
    return z[:, :w, :h].transpose(1, 2).contiguous()


def _box(d):
    return d.xmin, d.xmax, d.ymin, d.ymax


def _aos(f):
    """nine [n][h][w] -> [n][w][h][9]"""
    return torch.stack(f, dim=-1).transpose(1, 2).contiguous()


def _soa(a):
    """[n][w][h][9] -> nine [n][h][w]"""
    return [v.contiguous() for v in a.transpose(1, 2).unbind(-1)]


def exact(case, seed):
    c, kind = case, case["kind"]
    if kind == "step":
        w, h, *box = _geometry(c)
        masks, solid = _masks(h, w, box)
        post, rho, ux, uy = _collide(_soa(_states(w, h, 1, seed)), 1e-6, c["tau"])
        f = _stream(post, masks, solid)
        macro = torch.stack([v[0].t().reshape(-1) for v in (rho, ux, uy)])
        return dict(post=_aos(post)[0], state=_aos(f)[0], macro=macro, force=float(_force(f, box, c["tau"])[0]))
    if kind == "perturb":
        s = _states(c["width"], c["height"], c["nsnap"] + 1, seed)
        pre = torch.from_numpy(np.random.default_rng(seed).random(c["nsnap"])).cuda()
        mix = torch.tensordot(pre, s[1:], 1)
        wgt = s[0].norm() / mix.norm()
        return dict(state=(s[0] + 1e-3 * mix * wgt) / (1.0 + pre.sum() * 1e-3 * wgt))
    if kind == "warmup":
        d, _ = _single(c, seed)
        masks, solid = _masks(c["height"], c["width"], _box(d))
        f, drag = _soa(_states(c["width"], c["height"], 1, seed)), []
        for _ in range(c["steps"]):
            f = _stream(_collide(f, d.beta, d.tau)[0], masks, solid)
            drag.append(_force(f, _box(d), d.tau) * d.force_scale - d.force_shift)
        _, rho, ux, uy = _collide(f, d.beta, d.tau)
        flat = [v[0].t().reshape(-1).cpu().numpy() for v in (rho, ux, uy)]
        return dict(drag=torch.stack(drag, -1).cpu().numpy(), rho=flat[0], ux=flat[1], uy=flat[2],
                    state=_aos(f).reshape(-1).cpu().numpy())
    if kind == "adjoint":
        return _exact_adjoint(c, seed)
    return _exact_sampler(c, seed)


def _exact_adjoint(c, seed):
    """Reverse-mode differentiation of the plain forward, a few clones at a time."""
    d, r = _single(c, seed)
    box, (masks, solid) = _box(d), _masks(c["height"], c["width"], _box(d))
    part = max(1, 300_000 // (c["width"] * c["height"]) * 200 // max(c["steps"], 1))
    Js, grads = [], []
    for j in range(0, c["clones"], part):
        f0 = [v.requires_grad_() for v in _initial(r, box, 0, seed, j, min(part, c["clones"] - j))]
        f, J = f0, 0.0
        for _ in range(c["steps"]):
            f = _stream(_collide(f, d.beta, d.tau)[0], masks, solid)
            J = J + _force(f, box, d.tau) * d.force_scale - d.force_shift
        J = J * d.dt
        g = torch.autograd.grad(J.sum(), f0)
        Js.append(J.detach())
        grads.append(_aos([torch.where(solid, torch.zeros_like(v), v) for v in g]).reshape(len(J), -1))
    return dict(J=torch.cat(Js).cpu().numpy(), grad=torch.cat(grads).cpu().numpy())


def _exact_sampler(c, seed):
    drags, weights, rvals = [], [], []
    for i, (r, d) in enumerate(zip(_runs(c, seed), _descs(c, seed))):
        box = _box(d)
        masks, solid = _masks(r.height, r.width, box)
        part, series = max(1, 8_000_000 // (r.width * r.height)), []
        for j in range(0, r.nclones, part):
            n = min(part, r.nclones - j)
            f, out = _initial(r, box, i, seed, j, n), []
            field = 0.0
            if r.field_steps:
                field = torch.cat([_fields(r, i, d.seed, j + q, min(64, n - q)) for q in range(0, n, 64)])
            for t in range(c["steps"]):
                beta = d.beta * (1.0 + r.field_eps * field) if t < r.field_steps else d.beta
                f = _stream(_collide(f, beta, d.tau)[0], masks, solid)
                out.append(_force(f, box, d.tau, masks if d.drag_mode else None) * d.force_scale - d.force_shift)
            series.append(torch.stack(out, -1))
            del f
        F = torch.cat(series)
        wts = torch.exp(d.alpha * d.dt * F.sum(-1))
        drags.append(F)
        weights.append(wts)
        rvals.append(float(wts.mean()))
    F, wts = torch.cat(drags).cpu().numpy(), torch.cat(weights).cpu().numpy()
    if c["kind"] == "driver":
        return dict(labels=None, rvalue=rvals[0], weights=wts, copies_pre=None, copies_post=None, drag=F, state=None)
    return dict(rvalues=np.array(rvals)[:, None], drag=F[None], labels=None, weights=wts[None], state=None)
