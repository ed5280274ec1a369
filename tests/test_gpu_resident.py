"""Cluster-resident sweeps (wavefield in registers, one cluster per emitter group).

They evaluate every cell with the operations and rounding of the per-step kernels, so records,
wavefields, gradients and images must be equal bit for bit to those of the strip and tile kernels
(TOMO_RESIDENT=0) at every width class, with ragged widths and heights, single and many rows per
warp, checkpoints every 2 steps and full history, and for every cluster shape.  Against the FP64
oracle the parity bars of the other kernels hold.  A row that never arrives is a status.
"""
import numpy as np
import pytest

import oracle_lib as O
import tomo

pytestmark = pytest.mark.gpu

TOL_WAVE, TOL_GRAD = 1e-5, 1e-4


@pytest.fixture(scope="module", autouse=True)
def _lib(built_lib):
    return built_lib


def rel(a, b):
    a, b = np.asarray(a, np.float64), np.asarray(b, np.float64)
    return float(np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300))


def ring(nx, ny, nt, ns, gs, ckpt=0, sponge=8, **kw):
    return tomo.cfg_config(nx=nx, ny=ny, nt=nt, n_transducers=ns, group_size=gs, radius=min(0.42 * min(nx, ny), 0.5 * min(nx, ny) - 2.1),
                           cells_per_wavelength=8.0, sponge_width=sponge, ckpt_interval=ckpt, **kw)


def phantom(cfg):
    y, x = np.mgrid[0:cfg.ny, 0:cfg.nx]
    r2 = (x - 0.45 * cfg.nx) ** 2 + (y - 0.55 * cfg.ny) ** 2
    return (0.1 * (r2 < (0.15 * min(cfg.nx, cfg.ny)) ** 2)).astype(np.float32)


def sweep(cfg, fo):
    f0 = (0.4 * fo).astype(np.float32)
    with tomo.Context(cfg) as ctx:
        rec, last = ctx.forward(fo, u_last=True)
        dfg, _, r2 = ctx.gradient(f0, rec)
        f, g = f0.copy(), f0.copy()
        sched = tomo.schedule(omega=0.02, normalize=1)
        e = ctx.iterate(tomo.SIRT_CLASSIC, sched, 0, f, rec, fo).epsilon
        a = ctx.iterate(tomo.ART, sched, 0, g, rec, fo).epsilon
    return rec, last, dfg, np.float64(r2), f, g, np.float64(e), np.float64(a)


CASES = {
    "8x8 cells per lane 2, nt 4": dict(nx=16, ny=16, nt=4, ns=8, gs=4, sponge=2),
    "one block": dict(nx=64, ny=9, nt=60, ns=4, gs=2, sponge=2),
    "odd width and height, checkpoints of 2": dict(nx=61, ny=47, nt=91, ns=16, gs=4, ckpt=2, groups_per_pass=3),
    "65 columns (cells per lane 4)": dict(nx=65, ny=64, nt=120, ns=24, gs=4, ckpt=7),
    "sponge of one column": dict(nx=130, ny=97, nt=120, ns=24, gs=6, sponge=1, ckpt=11),
    "cells per lane 8": dict(nx=250, ny=130, nt=140, ns=40, gs=8, ckpt=25),
    "cells per lane 10": dict(nx=301, ny=233, nt=120, ns=40, gs=8),
    "cells per lane 12": dict(nx=322, ny=250, nt=90, ns=20, gs=5, ckpt=30),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_resident_matches_per_step_kernels(name, monkeypatch):
    cfg = ring(**CASES[name])
    fo = phantom(cfg)
    got = sweep(cfg, fo)
    monkeypatch.setenv("TOMO_RESIDENT", "0")
    want = sweep(cfg, fo)
    for k, (a, b) in enumerate(zip(got, want)):
        assert np.array_equal(a, b, equal_nan=True), (name, k, rel(a, b))
    assert np.abs(got[0]).max() > 0


# reference profile: rows between the paired ones even and odd in number, the smallest ring margin,
# non-square grids, right edges at each place of a lane, emission boxes around a corner
REF = {
    "64x60": dict(nx=64, ny=60, nt=150, ring_lo=8, ring_hi=50, group_size=24),
    "odd, checkpoints of 9": dict(nx=61, ny=53, nt=131, ring_lo=7, ring_hi=44, group_size=20, ckpt_interval=9,
                                  groups_per_pass=3),
    "least margin, checkpoints of 2": dict(nx=97, ny=98, nt=110, ring_lo=2, ring_hi=94, group_size=60, ckpt_interval=2),
    "smallest ring": dict(nx=22, ny=23, nt=90, ring_lo=8, ring_hi=11, group_size=4),
    "ring of two (per-step kernels)": dict(nx=24, ny=24, nt=60, ring_lo=10, ring_hi=12, group_size=4),
    "192": dict(nx=192, ny=192, nt=401, ring_lo=20, ring_hi=180, group_size=80),
    "195x130": dict(nx=195, ny=130, nt=160, ring_lo=11, ring_hi=117, group_size=100, ckpt_interval=33),
    "288": dict(nx=288, ny=288, nt=120, ring_lo=30, ring_hi=257, group_size=227),
}


@pytest.mark.parametrize("name", sorted(REF))
def test_reference_profile_matches_per_step_kernels(name, monkeypatch):
    cfg = tomo.ref_config(**REF[name])
    fo = 0.4 * phantom(cfg)
    got = sweep(cfg, fo)
    monkeypatch.setenv("TOMO_RESIDENT", "0")
    want = sweep(cfg, fo)
    for k, (a, b) in enumerate(zip(got, want)):
        assert np.array_equal(a, b, equal_nan=True), (name, k, rel(a, b))
    assert np.abs(got[0]).max() > 0


@pytest.mark.parametrize("shape", ["16,2", "13,2", "7,2"])
def test_every_reference_cluster_shape_gives_the_same_bits(shape, monkeypatch):
    cfg = tomo.ref_config(nx=118, ny=119, nt=140, ring_lo=13, ring_hi=104, group_size=91, ckpt_interval=21)
    fo = 0.4 * phantom(cfg)
    want = sweep(cfg, fo)
    monkeypatch.setenv("TOMO_RES_SHAPE", shape)
    got = sweep(cfg, fo)
    for k, (a, b) in enumerate(zip(got, want)):
        assert np.array_equal(a, b), (shape, k, rel(a, b))


@pytest.mark.parametrize("shape", ["16,1", "7,1", "16,2", "5,2", "4,4", "11,4"])
def test_every_cluster_shape_gives_the_same_bits(shape, monkeypatch):
    cfg = ring(nx=126, ny=111, nt=100, ns=30, gs=5, ckpt=13)
    fo = phantom(cfg)
    want = sweep(cfg, fo)
    monkeypatch.setenv("TOMO_RES_SHAPE", shape)
    got = sweep(cfg, fo)
    for k, (a, b) in enumerate(zip(got, want)):
        assert np.array_equal(a, b), (shape, k, rel(a, b))


def test_resident_matches_oracle():
    cfg = ring(nx=107, ny=94, nt=260, ns=24, gs=6, ckpt=19)
    fo = phantom(cfg)
    f0 = (0.4 * fo).astype(np.float32)
    rec_o = O.forward(cfg, fo.astype(np.float64))
    dfg_o, r2_o = O.gradient(cfg, f0.astype(np.float64), rec_o)
    with tomo.Context(cfg) as ctx:
        rec = ctx.forward(fo)
        dfg, _, r2 = ctx.gradient(f0, rec_o.astype(np.float32))
    assert rel(rec, rec_o) <= TOL_WAVE
    assert rel(dfg, dfg_o) <= TOL_GRAD
    assert abs(r2 - r2_o) <= 1e-5 * r2_o


@pytest.mark.parametrize("kind", [2, 3])
def test_resident_residual_noise(kind, monkeypatch):
    cfg = ring(nx=90, ny=70, nt=90, ns=20, gs=5)
    fo = phantom(cfg)
    outs = []
    for res in ("1", "0"):
        monkeypatch.setenv("TOMO_RESIDENT", res)
        with tomo.Context(cfg) as ctx:
            rec = ctx.forward(fo)
            ctx.set_residual_noise(kind, 0.1, 5)
            outs.append(ctx.gradient((0.5 * fo).astype(np.float32), rec)[0])
    assert np.array_equal(*outs)
    assert np.abs(outs[0]).max() > 0


@pytest.mark.parametrize("profile", ["ring", "reference"])
def test_row_that_never_arrives_is_a_status(profile, monkeypatch):
    """A cluster whose barriers expect bytes that never come gives up after the wait limit: the call
    returns TOMO_ERR_TIMEOUT, and a context made afterwards works."""
    if profile == "ring":
        cfg = ring(nx=96, ny=96, nt=80, ns=16, gs=8)
    else:
        cfg = tomo.ref_config(nx=64, ny=60, nt=60, ring_lo=8, ring_hi=50, group_size=42)
    fo = phantom(cfg)
    monkeypatch.setenv("TOMO_RES_SHAPE", "4,4" if profile == "ring" else "4,2")
    monkeypatch.setenv("TOMO_WAIT_LIMIT_NS", "2000000")
    monkeypatch.setenv("TOMO_TEST_UNDELIVERED_TX", "16")
    with tomo.Context(cfg) as ctx:
        with pytest.raises(tomo.TomoError) as e:
            ctx.forward(fo)
        assert e.value.status == tomo.ERR_TIMEOUT, e.value
    monkeypatch.delenv("TOMO_TEST_UNDELIVERED_TX")
    with tomo.Context(cfg) as ctx:
        rec = ctx.forward(fo)
    monkeypatch.setenv("TOMO_RESIDENT", "0")
    with tomo.Context(cfg) as ctx:
        assert np.array_equal(rec, ctx.forward(fo))


@pytest.mark.parametrize("cfg", [
    ring(nx=72, ny=64, nt=180, ns=24, gs=4), ring(nx=61, ny=47, nt=90, ns=16, gs=4), ring(nx=250, ny=190, nt=60, ns=60, gs=2),
    ring(nx=400, ny=396, nt=60, ns=16, gs=8), ring(nx=401, ny=397, nt=40, ns=16, gs=8),   # strips; per-cell
    tomo.ref_config(nx=61, ny=53, nt=100, ring_lo=7, ring_hi=44, group_size=2),
    tomo.ref_config(nx=340, ny=330, nt=40, ring_lo=20, ring_hi=300, group_size=280),     # per-cell
], ids=lambda c: f"{'reference' if c.profile == tomo.PROFILE_REF else 'ring'}-{c.nx}x{c.ny}")
def test_allocation_free_forward_has_the_same_bits(cfg):
    import ctypes as C

    import torch

    fo = (0.4 if cfg.profile == tomo.PROFILE_REF else 1.0) * phantom(cfg)
    with tomo.Context(cfg) as ctx:
        want = ctx.forward(fo)
    d_f = torch.from_numpy(fo.astype(np.float32)).cuda()
    d_rec = torch.full(want.shape, -1.0, device="cuda")
    torch.cuda.synchronize()
    for _ in range(2):
        assert tomo.lib().tomo_forward_noalloc(C.byref(cfg), C.c_void_p(d_f.data_ptr()), C.c_void_p(d_rec.data_ptr()),
                                               None) == tomo.OK
    torch.cuda.synchronize()
    assert np.array_equal(d_rec.cpu().numpy(), want)
