"""Performance cases of the wave-tomography engine: the calls a user makes, over the sizes they use.

Every case is one pass through a public entry point of the Python binding (the C ABI beneath it):
one reconstruction iteration, one forward solve, one rank's share of a gradient, one batch
iteration, one pass of the update network.  Inputs are made from the seed alone; measured records
are sums of delayed, attenuated pulses between every emitter of a group and every receiver plus 1 %
noise, which is what a scan of a weakly scattering object looks like.

`exact` restates each path in float64 with plain torch.
"""
import ctypes
import math
import os
import sys

import numpy as np
import torch

_PYTHON = os.path.join(os.getcwd(), "tomographic-image-reconstruction-algorithms_gb300", "python")
if _PYTHON not in sys.path:
    sys.path.insert(0, _PYTHON)

import tomo  # noqa: E402

DEV = "cuda:0"
METHODS = {"classic": tomo.SIRT_CLASSIC, "scaled": tomo.SIRT_SCALED, "norm": tomo.SIRT_NORM, "art": tomo.ART}


# ---- cases ---------------------------------------------------------------------------------------
def _ring(call, nx, ny, nt, ns, gs, radius, **kw):
    """A benchmark-profile problem: ns transducers on a circle, groups of gs."""
    c = dict(call=call, profile="ring", nx=nx, ny=ny, nt=nt, ns=ns, gs=gs, radius=radius, sponge=16, ckpt=0, per_pass=0,
             method="norm", step=0.02)
    c.update(kw)
    return c


def _square(call, n, nt, lo, hi, gs, **kw):
    """A reference-profile problem: transducers on a square ring between the sensor lines."""
    c = dict(call=call, profile="square", nx=n, ny=n, nt=nt, lo=lo, hi=hi, gs=gs, ckpt=0, per_pass=0, method="norm",
             step=0.02)
    c.update(kw)
    return c


def listed():
    return [
        # A forward solve in a caller that owns all device memory: the smallest call, many short steps.
        dict(_ring("forward_noalloc", 128, 128, 600, 32, 4, 50.0), name="noalloc-128"),
        # The 128 x 128 benchmark problem (3-disc phantom, uniform SIRT): small grid, latency per step.
        dict(_ring("iterate", 128, 128, 600, 32, 4, 50.0, method="classic", step=0.1), name="sirt-128"),
        # The 512 x 512 benchmark problem: weighted SIRT with checkpoints every 50 steps.
        dict(_ring("iterate", 512, 512, 2500, 256, 8, 220.0, ckpt=50), name="sirt-512"),
        # Sequential (Kaczmarz) updates: every pass carries one emitter group.
        dict(_ring("iterate", 256, 256, 2560, 128, 8, 110.0, ckpt=72, method="art"), name="art-256"),
        # One rank's share of the 2048 x 2048 problem's groups: wavefields far larger than the L2.
        dict(_ring("shard", 2048, 2048, 400, 512, 8, 950.0, per_pass=8, ckpt=200), name="shard-2048"),
        # A scan on a grid whose width and height divide nothing.
        dict(_ring("iterate", 301, 233, 1000, 60, 6, 100.0), name="sirt-301x233"),
        # The reference program's own problem (192 x 192, 401 steps, groups of 10), normalised SIRT.
        dict(_square("iterate", 192, 401, 20, 180, 10), name="ref-sirt-192"),
        # The reference's sequential driver on the same problem, groups of 20.
        dict(_square("iterate", 192, 401, 20, 180, 20, method="art"), name="ref-art-192"),
        # Data generation on the reference problem: forward solve and records only.
        dict(_square("forward", 192, 401, 20, 180, 10), name="ref-forward-192"),
        # Six phantoms of uneven sizes advanced together (the many-phantom workload's sizes).
        dict(call="batch", sizes="128,192,256,384,128,192", step=0.02, name="batch-6"),
        # The learned update's proposal for one 512 x 512 image.
        dict(call="net_forward", B=1, H=512, W=512, name="net-infer-512"),
        # One training gradient on the training set's batch shape.
        dict(call="net_grad", B=16, H=256, W=256, name="net-grad-16x256"),
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["iterate", "iterate", "iterate", "art", "shard", "forward", "noalloc", "square", "square",
                       "square-art", "square-forward", "batch", "net_forward", "net_grad"])
    if kind in ("iterate", "art", "shard", "forward", "noalloc"):
        nx = _logint(rng, 72, 2048 if kind == "shard" else 512 if kind == "noalloc" else 640)
        ny = min(max(64, int(nx * rng.uniform(0.75, 1.3))), 262144 // nx if kind == "noalloc" else 4096)
        if rng.random() < 0.5:                       # half of the widths a multiple of four, half as they come
            nx -= nx % 4
        m = min(nx, ny)
        gs = rng.choice([4, 5, 6, 8])
        ns = max(2, int(m * rng.uniform(0.2, 0.5)) // gs) * gs
        groups = ns // gs
        # steps: up to ten per cell of width, and no more cell updates than a third of the largest listed case
        share = rng.randint(1, min(8, groups)) if kind == "shard" else groups
        nt = min(int(m * rng.uniform(3.0, 10.0)), int(7e9 / (nx * ny * share)))
        if kind == "noalloc":
            nt = min(nt, 12000 // groups)
        if kind == "art":
            nt = min(nt, 40000 // groups)
        nt = max(120, nt)
        ckpt = rng.choice([0, 50, int(math.sqrt(2 * nt))])
        if ckpt == 0 and 4.0 * nx * ny * nt * share > 12e9:
            ckpt = int(math.sqrt(2 * nt))
        call = {"iterate": "iterate", "art": "iterate", "shard": "shard", "forward": "forward",
                "noalloc": "forward_noalloc"}[kind]
        method = "art" if kind == "art" else rng.choice(["classic", "scaled", "norm"])
        return _ring(call, nx, ny, nt, ns, gs, round(0.43 * m, 1), sponge=rng.choice([8, 12, 16]), ckpt=ckpt,
                     per_pass=share if kind == "shard" else 0, method=method, step=round(rng.uniform(0.01, 0.1), 3))
    if kind.startswith("square"):
        n = _logint(rng, 96, 288)
        lo = max(6, int(n * rng.uniform(0.08, 0.14)))
        hi = n - 1 - lo
        nt = int(n * rng.uniform(1.6, 2.4))
        gs = rng.choice([20, 32, 40] if kind == "square-art" else [10, 16, 20, 40, 80])
        call = "forward" if kind == "square-forward" else "iterate"
        return _square(call, n, nt, lo, hi, gs, method="art" if kind == "square-art" else rng.choice(["classic", "norm"]),
                       step=round(rng.uniform(0.01, 0.05), 3), ckpt=rng.choice([0, 0, 40]))
    if kind == "batch":
        k = rng.randint(2, 6)
        return dict(call="batch", sizes=",".join(str(rng.choice([96, 128, 160, 192, 256])) for _ in range(k)),
                    step=round(rng.uniform(0.01, 0.05), 3))
    W = 64 * _logint(rng, 1, 10)
    H = max(33, int(W * rng.uniform(0.5, 1.2)))
    return dict(call=kind, B=_logint(rng, 1, max(1, min(24, 1200000 // (H * W)))), H=H, W=W)


# ---- inputs --------------------------------------------------------------------------------------
def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(1000003 * int(seed) + 17)
    return g


def _uniform(g, n, lo, hi):
    return (lo + (hi - lo) * torch.rand(n, generator=g, device=DEV, dtype=torch.float64)).tolist()


def _phantom(c, g):
    """Eight ellipses of relative perturbation up to 0.12 inside the transducers, float32 on the GPU."""
    nx, ny = c["nx"], c["ny"]
    square = c["profile"] == "square"
    sup = 0.5 * (c["hi"] - c["lo"]) * 0.8 if square else 0.8 * c["radius"]
    y = torch.arange(ny, device=DEV, dtype=torch.float64)[:, None] - 0.5 * ny
    x = torch.arange(nx, device=DEV, dtype=torch.float64)[None, :] - 0.5 * nx
    f = torch.zeros(ny, nx, device=DEV, dtype=torch.float64)
    u = _uniform(g, 48, 0.0, 1.0)
    for e in range(8):
        a, b, th, val, rad, ang = u[6 * e:6 * e + 6]
        a, b = sup * (0.05 + 0.25 * a), sup * (0.05 + 0.25 * b)
        r = max(0.0, sup - max(a, b)) * math.sqrt(rad)
        dx, dy = x - r * math.cos(2 * math.pi * ang), y - r * math.sin(2 * math.pi * ang)
        ct, st = math.cos(math.pi * th), math.sin(math.pi * th)
        inside = ((dx * ct + dy * st) / a) ** 2 + ((dy * ct - dx * st) / b) ** 2 <= 1.0
        f = f + inside * ((0.01 + 0.04 * val) if square else 0.12 * (2 * val - 1))
    return f.float()


def _transducers(c):
    """0-based transducer cells (x, y) in ring order."""
    if c["profile"] == "ring":
        th = 2.0 * math.pi * np.arange(c["ns"]) / c["ns"]
        return (np.floor(0.5 * c["nx"] + c["radius"] * np.cos(th) + 0.5).astype(int),
                np.floor(0.5 * c["ny"] + c["radius"] * np.sin(th) + 0.5).astype(int))
    lo, hi = c["lo"], c["hi"]
    q = np.arange(1, hi - lo + 1)
    xs = np.concatenate([lo + q, 0 * q + hi, hi - q, 0 * q + lo])
    ys = np.concatenate([0 * q + hi, hi - q, 0 * q + lo, lo + q])
    return xs, ys


def _groups(c):
    return (c["ns"] if c["profile"] == "ring" else 4 * (c["hi"] - c["lo"])) // c["gs"]


def _receivers(c):
    """Receiver cell (x, y) per record channel and whether the channel has one."""
    if c["profile"] == "ring":
        x, y = _transducers(c)
        return x, y, np.ones(len(x), bool)
    n, lo, hi = c["nx"], c["lo"], c["hi"]
    t = np.arange(n)
    on = (t > lo) & (t < hi)
    return (np.concatenate([t, 0 * t + hi, t, 0 * t + lo]), np.concatenate([0 * t + hi, t, 0 * t + lo, t]),
            np.concatenate([on] * 4))


def _records(c, g):
    """Delayed, attenuated pulses from each group's emitters to every channel, and 1 % noise: float32 [G, nt, channels]."""
    ex, ey = _transducers(c)
    rx, ry, on = _receivers(c)
    ring = c["profile"] == "ring"
    dt = 0.5 if ring else 1500.0 * 3.3333e-07 / 1e-3         # cells a wave crosses per step
    t = dt * torch.arange(c["nt"], device=DEV, dtype=torch.float32)[:, None, None]
    rx, ry = (torch.tensor(v, device=DEV, dtype=torch.float32) for v in (rx, ry))
    live = torch.tensor(on, device=DEV)
    out = torch.empty(_groups(c), c["nt"], len(on), device=DEV, dtype=torch.float32)
    for k in range(_groups(c)):
        ids = range(k * c["gs"], (k + 1) * c["gs"], 1 if ring else max(1, c["gs"] // 8))
        px, py = (torch.tensor([float(v[i]) for i in ids], device=DEV) for v in (ex, ey))
        r = torch.hypot(rx[:, None] - px, ry[:, None] - py)
        p = (math.pi / 12.0) * (t - (0.99 * r + 18.0)) if ring else 0.25 * (t - (0.99 * r + 6.0))
        pulse = (1.0 - 2.0 * p * p) * torch.exp(-p * p) / torch.sqrt(torch.clamp(r, min=1.0))
        out[k] = (0.25 if ring else 0.5) * pulse.sum(-1)
    noise = torch.randn(out.shape, generator=g, device=DEV, dtype=torch.float32)
    return (out + 0.01 * out.std() * noise) * live


def _inputs(c, seed):
    g = _gen(seed)
    ft = _phantom(c, g)
    scale = 0.3 + 0.4 * _uniform(g, 1, 0.0, 1.0)[0]          # the image part-way through a reconstruction
    return ft, (scale * ft).contiguous(), (None if c["call"].startswith("forward") else _records(c, g))


def _config(c):
    kw = dict(ckpt_interval=c["ckpt"], groups_per_pass=c["per_pass"])
    if c["profile"] == "square":
        return tomo.ref_config(nx=c["nx"], ny=c["ny"], nt=c["nt"], group_size=c["gs"], ring_lo=c["lo"], ring_hi=c["hi"], **kw)
    return tomo.cfg_config(nx=c["nx"], ny=c["ny"], nt=c["nt"], n_transducers=c["ns"], group_size=c["gs"],
                           radius=c["radius"], sponge_width=c["sponge"], **kw)


def _phantoms(c):
    """The batch's problems: N x N grids, N / 2 transducers in groups of 8, 10 N steps."""
    out = []
    for n in (int(s) for s in c["sizes"].split(",")):
        out.append(_ring("iterate", n, n, 10 * n, n // 2, 8, 0.43 * n, ckpt=int(round(math.sqrt(20 * n))), step=c["step"]))
    return out


def _net_inputs(c, seed):
    """He-normal parameters, smooth features in [-1, 1], targets of a field update's size, a disc mask."""
    g = _gen(seed)
    parts = []
    for shape, sd in (((9, 16, 32), (2.0 / 27) ** 0.5), ((32,), 0.0), ((9, 32, 32), (2.0 / 288) ** 0.5), ((32,), 0.0),
                      ((9, 32, 32), (2.0 / 288) ** 0.5), ((32,), 0.0), ((9, 32, 32), (2.0 / 288) ** 0.5), ((32,), 0.0),
                      ((9, 32), 0.01 * (1.0 / 288) ** 0.5), ((1,), 0.0)):
        w = torch.randn(shape, generator=g, device=DEV) * (sd if sd else 0.01)
        if len(shape) == 3 and shape[1] == 16:
            w[:, 3:] = 0.0                                    # channels 3..15 are padding
        parts.append(w.reshape(-1))
    B, H, W = c["B"], c["H"], c["W"]
    low = torch.randn(B, 3, max(2, H // 8), max(2, W // 8), generator=g, device=DEV)
    feat = torch.tanh(torch.nn.functional.interpolate(low, size=(H, W), mode="bilinear")).contiguous()
    tgt = 0.02 * torch.randn(B, H, W, generator=g, device=DEV)
    y = torch.arange(H, device=DEV)[:, None] - 0.5 * H
    x = torch.arange(W, device=DEV)[None, :] - 0.5 * W
    mask = ((y / H) ** 2 + (x / W) ** 2 < 0.16).float().expand(B, H, W).contiguous()
    return torch.cat(parts), feat, tgt, mask


# ---- prepare and run -----------------------------------------------------------------------------
class _Problem:
    """A context with its records set, and the device buffers a program keeps beside it."""

    def __init__(self, c, seed):
        self.c, self.cfg = c, _config(c)
        self.ft, self.f0, rec = _inputs(c, seed)
        self.f = self.f0.clone()
        self.ctx = tomo.Context(self.cfg)
        self.stream = torch.cuda.ExternalStream(self.ctx.stream)
        if rec is not None:
            self.ctx.set_records(rec.cpu().numpy())
        self.sched = tomo.schedule(omega=c["step"], normalize=1)

    def restart(self):
        """The image of the iteration's start, on the context's stream."""
        self.stream.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(self.stream):
            self.f.copy_(self.f0)

    def join(self):
        torch.cuda.current_stream().wait_stream(self.stream)


def prepare(case, seed):
    call = case["call"]
    if call in ("iterate", "shard", "forward"):
        p = _Problem(case, seed)
        if call == "shard":
            p.out = torch.empty(case["per_pass"], case["ny"], case["nx"], device=DEV)
        if call == "forward":
            p.out = torch.empty(p.ctx.records_shape(), device=DEV)
        return p
    if call == "forward_noalloc":
        ft, _, _ = _inputs(case, seed)
        return {"call": call, "cfg": _config(case), "f": ft,
                "out": torch.empty(_groups(case), case["nt"], case["ns"], device=DEV)}
    if call == "batch":
        ps = [_Problem(c, 100 * seed + i) for i, c in enumerate(_phantoms(case))]
        return {"call": call, "ps": ps, "sched": tomo.schedule(omega=case["step"], normalize=1)}
    w, feat, tgt, mask = _net_inputs(case, seed)
    net = tomo.Net()
    net.set_params(w.cpu().numpy())
    return {"call": call, "net": net, "shape": (case["B"], case["H"], case["W"]), "feat": feat, "tgt": tgt, "mask": mask,
            "out": torch.empty(case["B"], case["H"], case["W"], device=DEV)}


def run(state):
    if isinstance(state, _Problem):
        p, c = state, state.c
        if c["call"] == "forward":
            p.stream.wait_stream(torch.cuda.current_stream())
            p.ctx.forward_device(p.ft.data_ptr(), p.out.data_ptr())
            p.join()
            return p.out
        p.restart()
        if c["call"] == "shard":
            r2 = p.ctx.gradient_groups_device(p.f.data_ptr(), 0, c["per_pass"])
            p.ctx.get_correlations_device(0, c["per_pass"], p.out.data_ptr())
            p.join()
            return {"corr": p.out, "resid_norm2": r2}
        st = p.ctx.iterate_device(METHODS[c["method"]], p.sched, 0, p.f.data_ptr(), 0, p.ft.data_ptr())
        p.join()
        return {"f": p.f, "epsilon": st.epsilon, "resid_norm2": st.resid_norm2}
    call = state["call"]
    if call == "forward_noalloc":
        st = tomo.lib().tomo_forward_noalloc(ctypes.byref(state["cfg"]), ctypes.c_void_p(state["f"].data_ptr()),
                                             ctypes.c_void_p(state["out"].data_ptr()),
                                             ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
        if st:
            raise tomo.TomoError(st, "tomo_forward_noalloc")
        return state["out"]
    if call == "batch":
        ps = state["ps"]
        for p in ps:
            p.restart()
        eps, _ = tomo.iterate_batch([p.ctx for p in ps], tomo.SIRT_NORM, state["sched"], 0, 1, [p.f.data_ptr() for p in ps],
                                    [p.ft.data_ptr() for p in ps])
        for p in ps:
            p.join()
        return {"f": [p.f for p in ps], "epsilon": eps}
    B, H, W = state["shape"]
    if call == "net_forward":
        state["net"].forward_device(state["feat"].data_ptr(), B, H, W, state["out"].data_ptr())
        return state["out"]
    g, loss = state["net"].grad_device(state["feat"].data_ptr(), state["tgt"].data_ptr(), state["mask"].data_ptr(), B, H, W)
    return {"grad": g, "loss": loss}


# ---- work ----------------------------------------------------------------------------------------
def work(case):
    """Inputs read once and outputs written once; one multiply or add per operation of the recurrences."""
    call = case["call"]
    if call == "batch":
        parts = [work(c) for c in _phantoms(case)]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    if call.startswith("net"):
        px = case["B"] * case["H"] * case["W"]
        macs = 9 * (3 * 32 + 3 * 32 * 32 + 32)
        if call == "net_forward":
            return {"bytes": 16.0 * px, "flops": 2.0 * macs * px}
        return {"bytes": 20.0 * px, "flops": 2.0 * (3 * macs - 9 * 3 * 32) * px}
    n = case["nx"] * case["ny"]
    groups = case["per_pass"] if call == "shard" else _groups(case)
    channels = case["ns"] if case["profile"] == "ring" else 4 * case["nx"]
    updates = float(groups) * n * (case["nt"] - 2)
    rec = 4.0 * groups * case["nt"] * channels
    fwd, adj = (11, 19) if case["profile"] == "ring" else (10, 21)
    if call.startswith("forward"):
        return {"bytes": 4.0 * n + rec, "flops": fwd * updates}
    out = 4.0 * n * groups if call == "shard" else 4.0 * n
    return {"bytes": rec + 8.0 * n + out, "flops": (fwd + adj) * updates}


# ---- float64 restatement -------------------------------------------------------------------------
DT, H0, WC, TAU, TT = (float(np.float32(v)) for v in (3.3333e-07, 0.001, 7.8540e+05, 4.0e-06, 8.1573e-06))


def _f64(t):
    return t.to(torch.float64)


def _pad(t):
    return torch.nn.functional.pad(t, (1, 1, 1, 1))


class _Ring64:
    """The benchmark profile: u+ = d (2u - u- + c lap u) + s, its exact adjoint and correlation."""

    def __init__(self, c):
        self.c = c
        nx, ny, w = c["nx"], c["ny"], c["sponge"]
        i = torch.arange(nx, device=DEV)[None, :].expand(ny, nx)
        j = torch.arange(ny, device=DEV)[:, None].expand(ny, nx)
        d = torch.minimum(torch.minimum(i, j), torch.minimum(nx - 1 - i, ny - 1 - j)).double()
        smax = float(np.float32(0.05))
        self.d = torch.where(d < w, 1.0 - smax * ((w - d) / w) ** 2, torch.ones_like(d))
        x, y = _transducers(c)
        cells = torch.tensor(y * nx + x, device=DEV)
        self.rcv = cells
        self.emit = cells[:_groups(c) * c["gs"]].reshape(_groups(c), c["gs"])
        self.mask = ((i - 0.5 * nx) ** 2 + (j - 0.5 * ny) ** 2 < (c["radius"] - 1.5) ** 2)
        self.src = []
        for n in range(c["nt"]):
            t = 0.5 * n - 18.0
            if t > 18.0:
                break
            a = (math.pi * t / 12.0) ** 2
            self.src.append(0.25 * (1.0 - 2.0 * a) * math.exp(-a))
        self.scale = 0.25

    def coef(self, f):
        return _pad(0.25 * (1.0 + f))

    @staticmethod
    def lap(p):
        q = p[:, 1:-1, 2:] + p[:, 1:-1, :-2]
        q += p[:, :-2, 1:-1]
        q += p[:, 2:, 1:-1]
        return q.sub_(p[:, 1:-1, 1:-1], alpha=4.0)

    def forward(self, cp, g0, ng, hist):
        c = self.c
        nx, ny = c["nx"], c["ny"]
        ci = cp[1:-1, 1:-1]
        hist[:2] = 0.0
        rows = torch.arange(ng, device=DEV)[:, None].expand(ng, c["gs"])
        em = self.emit[g0:g0 + ng]
        slots = hist.shape[0]
        rec = torch.zeros(ng, c["nt"], len(self.rcv), device=DEV, dtype=torch.float64)
        for k in range(1, c["nt"] - 1):
            u, up, un = hist[k % slots], hist[(k - 1) % slots], hist[(k + 1) % slots]
            v = self.lap(u).mul_(ci).add_(u[:, 1:-1, 1:-1], alpha=2.0).sub_(up[:, 1:-1, 1:-1]).mul_(self.d)
            if k < len(self.src):
                v.view(ng, -1).index_put_((rows, em), torch.full((), self.src[k], device=DEV, dtype=torch.float64),
                                          accumulate=True)
            un[:, 1:-1, 1:-1] = v
            rec[:, k + 1] = v.reshape(ng, ny * nx)[:, self.rcv]
        return rec

    def adjoint(self, f, cp, hist, rr, ng):
        c = self.c
        ny, nx = c["ny"], c["nx"]
        z1 = torch.zeros(ng, ny + 2, nx + 2, device=DEV, dtype=torch.float64)
        z2, corr = torch.zeros_like(z1), torch.zeros(ng, ny, nx, device=DEV, dtype=torch.float64)
        for m in range(c["nt"] - 1, 1, -1):
            z = self.lap(z1 * cp).add_(z1[:, 1:-1, 1:-1], alpha=2.0).sub_(z2[:, 1:-1, 1:-1])
            z.view(ng, -1)[:, self.rcv] += rr[:, m]
            z.mul_(self.d)
            corr.addcmul_(z, self.lap(hist[m - 1]))
            z2, z1 = z1, z2
            z1[:, 1:-1, 1:-1] = z
        return corr

    def interior(self, shape):
        return shape[0], shape[1] + 2, shape[2] + 2


class _Square64:
    """The reference profile: one-way edges with corner means, box emission, residual on the sensor lines."""

    def __init__(self, c):
        self.c = c
        n, lo, hi = c["nx"], c["lo"], c["hi"]
        self.mask = torch.zeros(n, n, device=DEV, dtype=torch.bool)
        self.mask[lo + 1:hi, lo + 1:hi] = True
        rx, ry, on = _receivers(c)
        self.on = torch.tensor(on, device=DEV)
        self.rcv = torch.tensor(np.where(on, ry * n + rx, 0), device=DEV)
        hh = np.float32(0.001) * np.float32(0.001)
        self.hh = H0 * H0
        self.scale = 1.0 / float(hh)
        x, y = _transducers(c)
        self.box = []
        for g in range(_groups(c)):
            a, b = g * c["gs"], (g + 1) * c["gs"] - 1
            self.box.append((min(x[a], x[b]), max(x[a], x[b]), min(y[a], y[b]), max(y[a], y[b])))

    def coef(self, f):
        return 1500.0 * torch.sqrt(1.0 + f)

    @staticmethod
    def corners(u):
        for j, jn in ((0, 1), (-1, -2)):
            for i, i_n in ((0, 1), (-1, -2)):
                u[:, j, i] = 0.5 * (u[:, jn, i] + u[:, j, i_n])

    def forward(self, v, g0, ng, hist):
        c = self.c
        r = v * DT / H0
        ri = r[1:-1, 1:-1]
        r2 = ri * ri
        hist[:2] = 0.0
        slots = hist.shape[0]
        inject = torch.zeros(ng, c["ny"], c["nx"], device=DEV, dtype=torch.float64)
        for k, (i0, i1, j0, j1) in enumerate(self.box[g0:g0 + ng]):
            inject[k, j0:j1 + 1, i0:i1 + 1] = 1.0
        inject = (inject * (v * v * DT * DT))[:, 1:-1, 1:-1]
        rec = torch.zeros(ng, c["nt"], len(self.rcv), device=DEV, dtype=torch.float64)
        edges = [((slice(None), 0, slice(1, -1)), (slice(None), 1, slice(1, -1)), (slice(None), 2, slice(1, -1))),
                 ((slice(None), -1, slice(1, -1)), (slice(None), -2, slice(1, -1)), (slice(None), -3, slice(1, -1))),
                 ((slice(None), slice(1, -1), 0), (slice(None), slice(1, -1), 1), (slice(None), slice(1, -1), 2)),
                 ((slice(None), slice(1, -1), -1), (slice(None), slice(1, -1), -2), (slice(None), slice(1, -1), -3))]
        for k in range(1, c["nt"] - 1):
            u, up, un = hist[k % slots], hist[(k - 1) % slots], hist[(k + 1) % slots]
            s = u[:, 1:-1, 2:] + u[:, 1:-1, :-2]
            s += u[:, :-2, 1:-1]
            s += u[:, 2:, 1:-1]
            s = s.mul_(r2).add_((2.0 - 4.0 * r2) * u[:, 1:-1, 1:-1]).sub_(up[:, 1:-1, 1:-1])
            if k + 1 <= 24:
                t = k * DT - TT
                s += inject * (math.cos(WC * t) * math.exp(-t * t / (2.0 * TAU * TAU)))
            un[:, 1:-1, 1:-1] = s
            for e, a, b in edges:
                q = r[e[1:]]
                un[e] = (2 - 2 * q - q * q) * u[e] + 2 * q * (1 + q) * u[a] - q * q * u[b] + (2 * q - 1) * up[e] - 2 * q * up[a]
            self.corners(un)
            rec[:, k + 1] = un.reshape(ng, -1)[:, self.rcv] * self.on
        return rec

    def adjoint(self, f, v, hist, rr, ng):
        c = self.c
        n, lo, hi = c["nx"], c["lo"], c["hi"]
        of = 1.0 + f
        z1 = torch.zeros(ng, n, n, device=DEV, dtype=torch.float64)
        z2, corr = torch.zeros_like(z1), torch.zeros_like(z1)
        A = 1500.0 * 1500.0 * DT * DT / self.hh
        b, t, sl = slice(lo + 1, hi), slice(1, -1), slice(None)
        for k in range(c["nt"] - 2, 0, -1):
            p = z1 * of
            z = z2                                            # z(k) overwrites z(k+2) cell by cell
            s = p[:, :-2, t] + p[:, 2:, t]
            s += p[:, t, :-2]
            s += p[:, t, 2:]
            s = s.sub_(p[:, t, t], alpha=4.0).mul_(A).add_(z1[:, t, t], alpha=2.0).sub_(z2[:, t, t])
            z[:, t, t] = s
            rk = rr[:, k] * (H0 * 1000.0)
            z[:, hi, b] = z[:, hi - 1, b] + rk[:, :n][:, b]
            z[:, lo, b] = z[:, lo + 1, b] + rk[:, 2 * n:3 * n][:, b]
            z[:, b, hi] = z[:, b, hi - 1] + rk[:, n:2 * n][:, b]
            z[:, b, lo] = z[:, b, lo + 1] + rk[:, 3 * n:][:, b]
            z[:, 0, t], z[:, -1, t] = z[:, 1, t], z[:, -2, t]
            z[:, t, 0], z[:, t, -1] = z[:, t, 1], z[:, t, -2]
            self.corners(z)
            u = torch.nn.functional.pad(hist[k][:, None], (1, 1, 1, 1), mode="replicate")[:, 0]
            lu = _Ring64.lap(u)
            self.corners(lu)
            corr.addcmul_(z, lu)
            z2, z1 = z1, z
        return corr

    def interior(self, shape):
        return shape


def _solver(c):
    return _Ring64(c) if c["profile"] == "ring" else _Square64(c)


def _chunk(c, groups):
    """Groups whose float64 history fits 16 GB together."""
    return max(1, min(groups, int(16e9 / (8.0 * (c["nx"] + 2) * (c["ny"] + 2) * c["nt"]))))


def _seconds(c, groups):
    """About how long the float64 sweep of this many groups takes."""
    per = 1 if c["method"] == "art" else _chunk(c, groups)
    ops = 22 if c["profile"] == "ring" else 75
    one = max(6e-6, per * c["nx"] * c["ny"] * 24.0 / 3e12)
    return math.ceil(groups / per) * c["nt"] * ops * one


def _sweep64(s, f, rec, g0, ng):
    """Raw correlations of groups g0 .. g0+ng-1 and their squared residual."""
    c = s.c
    cf = s.coef(f)
    hist = torch.zeros((c["nt"],) + tuple(s.interior((ng, c["ny"], c["nx"]))), device=DEV, dtype=torch.float64)
    rr = _f64(rec[g0:g0 + ng]) - s.forward(cf, g0, ng, hist)
    rr[:, :2] = 0.0
    if c["profile"] == "square":
        rr *= s.on
    return s.adjoint(f, cf, hist, rr, ng), float((rr * rr).sum())


def _update(s, f, d, step):
    m = float(d.abs()[s.mask].max())
    return torch.where(s.mask, f + (step / m if m > 0 else step) * d, f)


def _iterate64(c, seed):
    s = _solver(c)
    ft, f0, rec = _inputs(c, seed)
    ft, f = _f64(ft), _f64(f0)
    step, G, r2 = float(np.float32(c["step"])), _groups(c), 0.0
    if c["method"] == "art":
        for g in range(G):
            corr, e = _sweep64(s, f, rec, g, 1)
            r2 += e
            f = _update(s, f, corr[0] * s.scale / (1.0 + f), step)
    else:
        per, parts = _chunk(c, G), []
        for g in range(0, G, per):
            corr, e = _sweep64(s, f, rec, g, min(per, G - g))
            r2 += e
            parts.append(corr * s.scale / (1.0 + f))
        d = torch.cat(parts)
        if c["method"] == "norm":
            w = 1.0 / torch.sqrt(((d - d.sum(0) / G) ** 2).sum((1, 2)))
            d = (d * (w / w.sum())[:, None, None]).sum(0)
        else:
            d = d.sum(0) / (G if c["method"] == "scaled" else 1)
        f = _update(s, f, d, step)
    return f, 100.0 * float((f - ft).norm() / ft.norm()), r2


def _conv64(x, w, flip=False):
    """Sum over the nine taps of shifted x times w[tap]; flip: the transposed convolution."""
    B, H, W, _ = x.shape
    p = torch.nn.functional.pad(x, (0, 0, 1, 1, 1, 1))
    out = 0.0
    for tap in range(9):
        dy, dx = (2 - tap // 3, 2 - tap % 3) if flip else (tap // 3, tap % 3)
        out = out + p[:, dy:dy + H, dx:dx + W] @ (w[tap].T if flip else w[tap])
    return out


def _net64(case, seed):
    w, feat, tgt, mask = (_f64(t) for t in _net_inputs(case, seed))
    sizes, ws, o = [(9, 16, 32), (32,), (9, 32, 32), (32,), (9, 32, 32), (32,), (9, 32, 32), (32,), (9, 32, 1), (1,)], [], 0
    for s in sizes:
        n = int(np.prod(s))
        ws.append(w[o:o + n].reshape(s))
        o += n
    ys = [torch.nn.functional.pad(feat.permute(0, 2, 3, 1), (0, 13))]
    for l in range(4):
        ys.append(torch.relu(_conv64(ys[-1], ws[2 * l]) + ws[2 * l + 1]))
    out = _conv64(ys[4], ws[8])[..., 0] + ws[9]
    if case["call"] == "net_forward":
        return out
    e = (out - tgt) * mask
    msum = float(mask.sum())
    dz = (2.0 * e / msum)[..., None]
    B, H, W = case["B"], case["H"], case["W"]
    grads = []
    for l in range(4, -1, -1):
        p = torch.nn.functional.pad(ys[l], (0, 0, 1, 1, 1, 1))
        flat = dz.reshape(-1, dz.shape[-1])
        gw = torch.stack([p[:, t // 3:t // 3 + H, t % 3:t % 3 + W].reshape(-1, p.shape[-1]).T @ flat for t in range(9)])
        grads = [gw.reshape(-1), flat.sum(0)] + grads
        if l:
            dz = _conv64(dz, ws[2 * l], flip=True) * (ys[l] > 0)
    return {"grad": torch.cat(grads).cpu().numpy(), "loss": float((e * e).sum()) / msum}


def exact(case, seed):
    call = case["call"]
    if call.startswith("net"):
        return _net64(case, seed)
    if call == "batch":
        cs = _phantoms(case)
        if sum(_seconds(c, _groups(c)) for c in cs) > 20:
            return None
        got = [_iterate64(c, 100 * seed + i) for i, c in enumerate(cs)]
        return {"f": [g[0] for g in got], "epsilon": np.array([[g[1]] for g in got])}
    groups = case["per_pass"] if call == "shard" else _groups(case)
    if _seconds(case, groups) > 20:
        return None
    if call.startswith("forward"):
        s = _solver(case)
        f = _f64(_inputs(case, seed)[0])
        per, out = _chunk(dict(case, nt=3), groups), []
        for g in range(0, groups, per):
            ng = min(per, groups - g)
            hist = torch.zeros((3,) + tuple(s.interior((ng, case["ny"], case["nx"]))), device=DEV, dtype=torch.float64)
            out.append(s.forward(s.coef(f), g, ng, hist))
        return torch.cat(out)
    if call == "shard":
        s = _solver(case)
        _, f0, rec = _inputs(case, seed)
        per, parts, r2 = _chunk(case, groups), [], 0.0
        for g in range(0, groups, per):
            corr, e = _sweep64(s, _f64(f0), rec, g, min(per, groups - g))
            parts.append(corr)
            r2 += e
        return {"corr": torch.cat(parts), "resid_norm2": r2}
    f, eps, r2 = _iterate64(case, seed)
    return {"f": f, "epsilon": eps, "resid_norm2": r2}
