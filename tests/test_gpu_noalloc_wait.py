"""A row that never arrives in the allocation-free forward.

The call returns before its kernel runs, so a wait that runs out cannot be its status: every record of the
group must then be NaN instead of a record that stops, and the next call must be right again.  The rows are
withheld as in the contexts' test: barriers that expect bytes which never come, and a short limit.
"""
import ctypes as C

import numpy as np
import pytest

import tomo

pytestmark = pytest.mark.gpu

CASES = {
    # two groups on clusters of 16 blocks; the reference profile's rows come in pairs
    "ring": lambda: tomo.cfg_config(nx=96, ny=96, nt=80, n_transducers=16, group_size=8, radius=40.0, cells_per_wavelength=8.0,
                                    sponge_width=8),
    "reference": lambda: tomo.ref_config(nx=64, ny=60, nt=60, ring_lo=8, ring_hi=50, group_size=42),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_row_that_never_arrives_leaves_nan(built_lib, name, monkeypatch):
    import torch

    cfg = CASES[name]()
    y, x = np.mgrid[0:cfg.ny, 0:cfg.nx]
    fo = (0.05 * ((x - 0.5 * cfg.nx) ** 2 + (y - 0.5 * cfg.ny) ** 2 < 100)).astype(np.float32)
    d_f = torch.from_numpy(fo).cuda()
    d_rec = torch.zeros((tomo.n_groups(cfg), cfg.nt, tomo.n_channels(cfg)), device="cuda")

    def call():
        torch.cuda.synchronize()
        st = built_lib.tomo_forward_noalloc(C.byref(cfg), C.c_void_p(d_f.data_ptr()), C.c_void_p(d_rec.data_ptr()), None)
        assert st == tomo.OK
        torch.cuda.synchronize()
        return d_rec.cpu().numpy()

    monkeypatch.setenv("TOMO_WAIT_LIMIT_NS", "2000000")
    monkeypatch.setenv("TOMO_TEST_UNDELIVERED_TX", "16")
    assert np.isnan(call()).all()
    monkeypatch.delenv("TOMO_WAIT_LIMIT_NS")
    monkeypatch.delenv("TOMO_TEST_UNDELIVERED_TX")
    got = call()
    with tomo.Context(cfg) as ctx:
        want = ctx.forward(fo)
    assert np.array_equal(got, want) and np.abs(want).max() > 0


def test_context_names_the_row(built_lib, monkeypatch):
    """The contexts' message covers both kinds of wait: a resident sweep has no TMA copy."""
    cfg = CASES["ring"]()
    monkeypatch.setenv("TOMO_WAIT_LIMIT_NS", "2000000")
    monkeypatch.setenv("TOMO_TEST_UNDELIVERED_TX", "16")
    monkeypatch.setenv("TOMO_RES_SHAPE", "16,1")
    with tomo.Context(cfg) as ctx:
        with pytest.raises(tomo.TomoError) as e:
            ctx.forward(np.zeros((cfg.ny, cfg.nx), np.float32))
    assert e.value.status == tomo.ERR_TIMEOUT and "row did not arrive" in str(e.value), e.value
