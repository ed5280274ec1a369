"""Streamed sweeps: several time steps per launch on grids that do not stay on chip.

They evaluate every cell with the operations and rounding of the per-step kernels, so records,
wavefields, gradients and images must be equal bit for bit to those of the strip, tile and per-cell
kernels (TOMO_RESIDENT=0).  TOMO_STREAM=1 streams grids of any size, which lets small ones reach the
edges: one strip and several, their last with one column, bands of one row, segments of every length
mod 4, more receivers on a strip than it keeps in shared memory, no sponge.
"""
import numpy as np
import pytest

import tomo

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _lib(built_lib):
    return built_lib


def ring(nx, ny, nt, ns, gs, ckpt=0, sponge=8, **kw):
    return tomo.cfg_config(nx=nx, ny=ny, nt=nt, n_transducers=ns, group_size=gs, radius=min(0.42 * min(nx, ny), 0.5 * min(nx, ny) - 2.1),
                           cells_per_wavelength=8.0, sponge_width=sponge, ckpt_interval=ckpt, **kw)


def phantom(cfg):
    y, x = np.mgrid[0:cfg.ny, 0:cfg.nx]
    r2 = (x - 0.45 * cfg.nx) ** 2 + (y - 0.55 * cfg.ny) ** 2
    return (0.1 * (r2 < (0.15 * min(cfg.nx, cfg.ny)) ** 2)).astype(np.float32)


def sweep(cfg, noise=0):
    fo = phantom(cfg)
    f0 = (0.4 * fo).astype(np.float32)
    with tomo.Context(cfg) as ctx:
        rec, last = ctx.forward(fo, u_last=True)
        if noise:
            ctx.set_residual_noise(noise, 0.1, 5)
        dfg, _, r2 = ctx.gradient(f0, rec)
        f, g = f0.copy(), f0.copy()
        sched = tomo.schedule(omega=0.02, normalize=1)
        e = ctx.iterate(tomo.SIRT_CLASSIC, sched, 0, f, rec, fo).epsilon
        a = ctx.iterate(tomo.ART, sched, 0, g, rec, fo).epsilon
    return rec, last, dfg, np.float64(r2), f, g, np.float64(e), np.float64(a)


CASES = {
    "nt 4": (dict(nx=16, ny=16, nt=4, ns=8, gs=4, sponge=2), 0),
    "nt 5": (dict(nx=60, ny=11, nt=5, ns=4, gs=2, sponge=2), 0),
    "one column in the last strip": (dict(nx=113, ny=47, nt=91, ns=16, gs=4, ckpt=2, groups_per_pass=3), 0),
    "one column in the adjoint's last strip": (dict(nx=57, ny=130, nt=92, ns=16, gs=4, ckpt=3), 0),
    "one row in the last band": (dict(nx=112, ny=121, nt=93, ns=16, gs=16, ckpt=5), 0),
    "no sponge": (dict(nx=131, ny=97, nt=94, ns=24, gs=6, sponge=0, ckpt=11), 0),
    "300 receivers on two strips": (dict(nx=140, ny=150, nt=80, ns=300, gs=100, ckpt=13), 0),
    "residual noise": (dict(nx=150, ny=90, nt=80, ns=20, gs=5, ckpt=30), 3),
    "odd width": (dict(nx=403, ny=390, nt=70, ns=40, gs=8), 0),
    "many groups": (dict(nx=230, ny=228, nt=70, ns=64, gs=1, ckpt=17), 0),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_streamed_matches_per_step_kernels(name, monkeypatch):
    args, noise = CASES[name]
    cfg = ring(**args)
    monkeypatch.setenv("TOMO_STREAM", "1")
    got = sweep(cfg, noise)
    monkeypatch.delenv("TOMO_STREAM")
    monkeypatch.setenv("TOMO_RESIDENT", "0")
    want = sweep(cfg, noise)
    for k, (a, b) in enumerate(zip(got, want)):
        assert np.array_equal(a, b, equal_nan=True), (name, k)
    assert np.abs(got[0]).max() > 0


def test_choice_keeps_the_bits(monkeypatch):
    """A grid too large for the chip and a sweep long enough for the trial: whichever is chosen."""
    cfg = ring(nx=444, ny=440, nt=120, ns=32, gs=8, ckpt=25)
    got = sweep(cfg)
    monkeypatch.setenv("TOMO_STREAM", "0")
    want = sweep(cfg)
    for k, (a, b) in enumerate(zip(got, want)):
        assert np.array_equal(a, b, equal_nan=True), k


def test_least_memory_falls_back(monkeypatch):
    """A limit that holds one group of the per-step kernels but not the streamed one's extra slices:
    the call still runs, with the same bits."""
    cfg = ring(nx=600, ny=600, nt=24, ns=8, gs=8, ckpt=2)
    want = sweep(cfg)
    outs = 0
    for mb in range(64, 160, 2):
        cfg.mem_limit_mb = mb
        monkeypatch.setenv("TOMO_STREAM", "0")
        try:
            tomo.Context(cfg).close()
        except tomo.TomoError:
            continue
        monkeypatch.delenv("TOMO_STREAM")
        got = sweep(cfg)
        for k, (a, b) in enumerate(zip(got, want)):
            assert np.array_equal(a, b, equal_nan=True), (mb, k)
        outs += 1
        break
    assert outs == 1


@pytest.mark.parametrize("cfg", [
    ring(nx=512, ny=512, nt=60, ns=16, gs=4),                        # the largest: framed slices fill the array
    ring(nx=449, ny=451, nt=61, ns=150, gs=50, sponge=0),            # as it comes; one step left over
    ring(nx=700, ny=371, nt=62, ns=24, gs=8), ring(nx=301, ny=700, nt=63, ns=24, gs=8),
    ring(nx=250, ny=1000, nt=5, ns=8, gs=8), ring(nx=400, ny=388, nt=4, ns=8, gs=4),
    ring(nx=9, ny=1030, nt=20, ns=2, gs=1, sponge=2),                # more rows than tables: per-cell kernels
    ring(nx=13000, ny=20, nt=20, ns=4, gs=1, sponge=2),              # the frame does not fit: per-cell kernels
], ids=lambda c: f"{c.nx}x{c.ny}")
def test_allocation_free_forward_streams(cfg, monkeypatch):
    import ctypes as C

    import torch

    fo = phantom(cfg)
    monkeypatch.setenv("TOMO_RESIDENT", "0")
    with tomo.Context(cfg) as ctx:
        want = ctx.forward(fo)
    monkeypatch.delenv("TOMO_RESIDENT")
    d_f = torch.from_numpy(fo).cuda()
    d_rec = torch.full(want.shape, -1.0, device="cuda")
    torch.cuda.synchronize()
    for _ in range(2):
        assert tomo.lib().tomo_forward_noalloc(C.byref(cfg), C.c_void_p(d_f.data_ptr()), C.c_void_p(d_rec.data_ptr()),
                                               None) == tomo.OK
    torch.cuda.synchronize()
    assert np.array_equal(d_rec.cpu().numpy(), want)
    assert np.abs(want).max() > 0
