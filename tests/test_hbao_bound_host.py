"""What decides an ambient-occlusion byte from the kernel's estimate: the bound of
the estimated sum, and poly_pow's error, which is below half of the slack given
to it at every exponent."""
import numpy as np
import pytest

from oracle import hbao as H
from test_native_host import test_native as _run


def test_bound_of_the_estimated_sum(tmp_path):
    _run("hbao_bound_test", tmp_path)


@pytest.mark.parametrize("e", [0.01, 0.1, 0.732, 1.0, 1.1, 2.0, 3.0, 10.0, 100.0, 1e4])
def test_error_of_poly_pow(e):
    rng = np.random.default_rng(0)
    a = np.concatenate([rng.uniform(0, 1, 400000), 1 - 0.1 * rng.uniform(0, 1, 100000) ** 4,
                        np.exp(-rng.uniform(0, 80, 100000))]).astype(np.float32)
    a = a[(a > 0) & (a <= 1)]
    e = np.float32(e)
    off = np.abs(H.poly_pow(a, e).astype(np.float64) - a.astype(np.float64) ** np.float64(e)).max()
    assert 2 * off < 5e-7 + 3e-7 * e
