"""The range over which the reference-profile adjoint divides by h^2 with a product and one correction.

The kernel scales by 2^64, multiplies by 1 / h^2 (10^6) and corrects once; lanes with a value above a bound divide
instead.  Nothing may overflow at or below that bound: the quotient must be the correctly rounded one up to it, at
both signs, with a sample of significands at every exponent.
"""
import os
import re

import numpy as np

import test_div_cpu as D

SOURCE = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "tomographic-image-reconstruction-algorithms_gb300",
                      "csrc", "resident_ref.cuh")


def test_quotient_up_to_the_bound():
    exponent = int(re.search(r"if \(most > 0x1p(\d+)f\)", open(SOURCE).read()).group(1))
    rng = np.random.default_rng(2)
    frac = np.concatenate([[0, 1, (1 << 23) - 1], rng.integers(0, 1 << 23, 2000)]).astype(np.uint32)
    with np.errstate(over="ignore", invalid="ignore"):
        for e in range(-20, exponent):
            x = (frac | np.uint32((127 + e) << 23)).view(np.float32)
            x = np.concatenate([x, -x])
            got, HH, _ = D.quotient(x)
            assert np.array_equal(got, x / HH), e
        x = np.array([2.0 ** exponent], np.float32)
        got, HH, _ = D.quotient(x)
        assert np.array_equal(got, x / HH)
