"""A context's kernel trials leave correlations alone that an earlier pass has left there.

Kernels are chosen when a pass of one group, or of several, first runs, which can be in the middle of a
gradient (a last pass of one group) or between two calls whose correlations stay in the context (group
ranges of unequal lengths).  Trials also write residual records, which a pass must find as if there had been none.  The first results of a fresh context must equal its second ones, and those of
a context that keeps to the per-step kernels, bit for bit.  Grids: one that stays on chip; too large for it, a width that
is a multiple of four and enough steps for the trials; passes of several groups below and above the 32 MiB
from which they are streamed without a trial (above it, the per-step kernels' own trials come with the
first pass of one group, and run on as many groups as a pass holds).
"""
import numpy as np
import pytest

import tomo

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _lib(built_lib):
    return built_lib


def ring(n, groups, per_pass, ckpt):
    # a small ring: echoes of the disc inside it return within the sweep
    return tomo.cfg_config(nx=n, ny=n - 4, nt=96, n_transducers=2 * groups, group_size=2, radius=20.0, cells_per_wavelength=8.0,
                           sponge_width=8, ckpt_interval=ckpt, groups_per_pass=per_pass)


SMALL = ring(448, 9, 4, 0)
CASES = {
    "passes of 4, 4 and 1": SMALL,
    "checkpoints": ring(448, 9, 4, 15),
    "timed memory plan": ring(448, 9, 4, -1),
    "held on chip": ring(128, 9, 4, 15),
    "above 32 MiB a slice": ring(1024, 9, 8, 12),
    "above 32 MiB a slice, full history": ring(1024, 9, 8, 0),
}


def fields(cfg):
    y, x = np.mgrid[0:cfg.ny, 0:cfg.nx]
    fo = (0.1 * ((x - 0.5 * cfg.nx + 3) ** 2 + (y - 0.5 * cfg.ny - 2) ** 2 < 121)).astype(np.float32)
    return fo, (0.4 * fo).astype(np.float32)


def records(cfg, fo):
    with tomo.Context(cfg) as ctx:
        return ctx.forward(fo)


@pytest.mark.parametrize("name", sorted(CASES))
def test_first_gradient_equals_the_second(name, monkeypatch):
    cfg = CASES[name]
    fo, f0 = fields(cfg)
    rec = records(cfg, fo)
    with tomo.Context(cfg) as ctx:
        first, d1, r1 = ctx.gradient(f0, rec)
        second, d2, r2 = ctx.gradient(f0, rec)
    assert [g for g in range(len(first)) if not np.array_equal(first[g], second[g])] == []
    assert np.array_equal(d1, d2) and r1 == r2
    assert all(np.abs(g).max() > 0 for g in first)
    monkeypatch.setenv("TOMO_STREAM", "0")
    monkeypatch.setenv("TOMO_RESIDENT", "0")
    with tomo.Context(cfg) as ctx:
        want, d, r = ctx.gradient(f0, rec)
    assert np.array_equal(first, want) and np.array_equal(d1, d) and r1 == r


@pytest.mark.parametrize("method", [tomo.SIRT_CLASSIC, tomo.SIRT_NORM])
def test_first_iteration(method, monkeypatch):
    cfg = SMALL
    fo, f0 = fields(cfg)
    rec = records(cfg, fo)
    sched = tomo.schedule(omega=0.02, normalize=1)
    out = []
    for stream in ("", "0"):
        monkeypatch.setenv("TOMO_STREAM", stream)
        with tomo.Context(cfg) as ctx:
            f = f0.copy()
            e = [ctx.iterate(method, sched, k, f, rec, fo).epsilon for k in range(2)]
            out.append((f, e))
    assert np.array_equal(out[0][0], out[1][0]) and out[0][1] == out[1][1]


@pytest.mark.parametrize("ranges", [((0, 4), (4, 1)), ((0, 1), (1, 4)), ((1, 4), (0, 1)), ((4, 1), (0, 4))], ids=str)
@pytest.mark.parametrize("big", [False, True], ids=["448", "1024"])
def test_group_ranges_keep_earlier_correlations(ranges, big):
    import torch

    cfg = ring(1024, 9, 8, 12) if big else SMALL
    if big:   # a pass of eight groups of 1024 x 1020 is above the 32 MiB
        ranges = tuple((a * 2 if a > 1 else a, 8 if n == 4 else n) for a, n in ranges)
    fo, f0 = fields(cfg)
    rec = records(cfg, fo)
    d_f = torch.from_numpy(f0).cuda()
    groups = sum(n for _, n in ranges)

    def correlations(ctx):
        for g0, ng in ranges:
            ctx.gradient_groups_device(d_f.data_ptr(), g0, ng)
        out = torch.empty((groups,) + f0.shape, device="cuda")
        torch.cuda.synchronize()
        ctx.get_correlations_device(0, groups, out.data_ptr())
        ctx.synchronize()
        return out.cpu().numpy()

    with tomo.Context(cfg) as ctx:
        ctx.set_records(rec)
        first, second = correlations(ctx), correlations(ctx)
    assert [g for g in range(groups) if not np.array_equal(first[g], second[g])] == []
    assert all(np.abs(g).max() > 0 for g in first)
