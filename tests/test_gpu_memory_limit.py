"""A context stays within its memory limit.

On a grid that is not held on chip the streamed sweeps keep a framed coefficient and sponge map beside the
plan's buffers, 134 MB at 4096 x 4096.  The limits run from too little for any plan past the one from which
the sweeps are streamed; the plan must count everything at each.
"""
import pytest

import tomo

pytestmark = pytest.mark.gpu


def test_device_bytes_stay_within_the_limit(built_lib):
    cfg = tomo.cfg_config(nx=4096, ny=4096, nt=8, n_transducers=8, group_size=8, radius=1000.0, ckpt_interval=2)
    sizes = []
    for mb in range(1400, 2120, 40):
        cfg.mem_limit_mb = mb
        try:
            with tomo.Context(cfg) as ctx:
                sizes.append((mb, ctx.info.device_bytes))
        except tomo.TomoError as e:
            assert e.status == tomo.ERR_OOM and not sizes, (mb, e)   # refused below the least, never above it
    assert [(mb, b) for mb, b in sizes if b > mb << 20] == []
    assert len(sizes) < 18 and sizes[-1][1] > sizes[0][1] + (300 << 20)   # both kinds of plan were seen
