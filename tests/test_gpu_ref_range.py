"""Reference-profile gradients of records at every magnitude, held on chip against the per-step kernels.

The adjoint wave scales with the records; where its values pass the range in which the on-chip sweep replaces the
division by h^2, it must divide.  Same bits as the per-step kernels from records far too small to 10^36.  Above,
where values pass 8.5 x 10^37, the per-step kernels' separate product 4 z is infinite and the fused one is not.
"""
import numpy as np
import pytest

import tomo

pytestmark = pytest.mark.gpu


def test_records_of_every_magnitude(built_lib, monkeypatch):
    cfg = tomo.ref_config(nx=61, ny=53, nt=90, ring_lo=7, ring_hi=44, group_size=20)
    y, x = np.mgrid[0:cfg.ny, 0:cfg.nx]
    fo = (0.04 * ((x - 25) ** 2 + (y - 25) ** 2 < 100)).astype(np.float32)
    with tomo.Context(cfg) as ctx:
        rec = ctx.forward(fo)
    rec /= np.abs(rec).max()
    scales = [10.0 ** k for k in range(-44, 38, 2)]
    out = []
    for res in ("1", "0"):
        monkeypatch.setenv("TOMO_RESIDENT", res)
        with tomo.Context(cfg) as ctx:
            out.append([ctx.gradient(np.zeros_like(fo), (rec * s).astype(np.float32))[0] for s in scales])
    wrong = [s for s, a, b in zip(scales, *out) if not np.array_equal(a, b, equal_nan=True)]
    assert wrong == []
    assert sum(bool(np.isfinite(a).all() and np.abs(a).max() > 1e12) for a in out[0]) >= 3   # large and finite ones among them
