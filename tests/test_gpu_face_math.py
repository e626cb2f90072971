"""What stands in for IEEE divisions and square roots on the float64 path, against
the IEEE operations: the faces' reciprocals and roots (one third-order step from the
hardware approximation) and the update's quotients."""
import ctypes as C

import numpy as np
import pytest
import torch

from astrofd_b200 import _lib

pytestmark = pytest.mark.gpu

RCP, RSQ, ROOT, QUOT = range(4)


def _device(op, x, d=1.0):
    x = np.ascontiguousarray(x, dtype=np.float64)
    xd = torch.from_numpy(x).cuda()
    yd = torch.empty_like(xd)
    assert _lib.load().astro_debug_math_f64(op, C.c_void_p(xd.data_ptr()), d, C.c_void_p(yd.data_ptr()),
                                            x.size, None) == 0
    torch.cuda.synchronize()
    return yd.cpu().numpy()


def _values(lo, hi, n, seed):
    """|x| over [2^lo, 2^hi), every power of two and its neighbours among them, and
    mantissas close to 1 and 2."""
    r = np.random.default_rng(seed)
    p = 2.0 ** np.arange(lo, hi)
    x = np.concatenate([2.0 ** r.uniform(lo, hi, n), p, np.nextafter(p, 0) if lo > -1022 else p,
                        np.nextafter(p, np.inf), 1.0 + 2.0 ** -r.uniform(1, 52, n // 8),
                        2.0 - 2.0 ** -r.uniform(1, 51, n // 8), r.uniform(0, 1, n)])
    return x[x >= 2.0 ** lo]


def _within(y, ref, ulps):
    # the reference is itself rounded: half an ulp of the bound
    return np.all(np.abs(y - ref) <= ulps * np.spacing(np.abs(ref)))


def test_reciprocal():
    x = _values(-1021, 1021, 1 << 19, 1)
    x = np.concatenate([x, -x])
    assert _within(_device(RCP, x), 1.0 / x, 2)


def test_reciprocal_root():
    x = _values(-1022, 1023, 1 << 19, 2)
    assert _within(_device(RSQ, x), 1.0 / np.sqrt(x), 2)


def test_root():
    x = _values(-960, 1023, 1 << 19, 3)  # above 1e-290
    assert _within(_device(ROOT, x), np.sqrt(x), 2)
    small = np.array([0.0, 5e-324, 1e-300, 9e-291])
    y = _device(ROOT, small)
    assert np.all(y >= 0.0) and np.all(y <= 1e-145) and y[0] == 0.0


def test_out_of_range_is_not_finite():
    """What sends a face to the general evaluation."""
    bad = np.array([0.0, -0.0, np.inf, -np.inf, np.nan, 5e-324, 1e-310])
    assert not np.isfinite(_device(RCP, bad)).any()
    assert not np.isfinite(_device(RSQ, np.concatenate([bad, [-1.0, -1e-300, -1e300]]))).any()
    assert not np.isfinite(_device(ROOT, np.array([np.inf, np.nan]))).any()
    # the reciprocal's own result would be subnormal
    assert np.array_equal(_device(RCP, np.array([1.7e308, -1.7e308])), [0.0, -0.0])


@pytest.mark.parametrize("d", [1.0 / 128, 1.0 / 61, 0.1, 1.0, 3.0, 1e-5, np.nextafter(1.0, 2), 2.0 - 2.0 ** -52])
def test_quotient_is_the_ieee_quotient(d):
    r = np.random.default_rng(int(d * 1e6))
    x = np.concatenate([r.standard_normal(1 << 19), 10.0 ** r.uniform(-200, 200, 1 << 19), [0.0, -0.0, d, 2 * d]])
    assert np.array_equal(_device(QUOT, x, float(d)), x / d)
