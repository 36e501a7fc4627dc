"""The plain form's own FP64 reciprocal, reciprocal square root and
exponential (csrc/vx_pairs.cu) against 64-bit mantissas on the host, over every
exponent of their ranges and at the ends.

Bounds, in units of u = 2^-53 relative to the value.  With seeds good to 2^-20:
the reciprocal's cubic step leaves e^3 = 2^-60 and the rounding of its last sum,
1.01 u; the root's residual e = 1 - x y^2 is off by u from the rounding of x y,
which counts half, its step leaves 5/16 (2^-19)^3 = 2^-58.7, 1.6 u with the last
rounding.  The exponential has the table's rounding and the last sum's, u each,
four more of its polynomial and product at most 0.011 of it, and 2^-58 left out:
2.1 u."""
import ctypes as C

import numpy as np
import pytest
import torch

from vortex_b200 import native as N

pytestmark = pytest.mark.gpu

RCP, RSQRT, EXP = 0, 1, 2


def device(which, x):
    dx = torch.from_numpy(x).cuda()
    out = torch.empty_like(dx)
    assert N.lib().vx_eval_fp64(C.c_int(which), C.c_void_p(dx.data_ptr()), C.c_void_p(out.data_ptr()),
                                C.c_int64(len(x))) == 0
    return out.cpu().numpy()


def every_exponent(lo, hi, seed):
    """For each exponent in [lo, hi]: its first, second, middle and last
    values, and random ones."""
    rng = np.random.default_rng(seed)
    u = 2.0 ** -52
    m = np.concatenate([[1.0, 1.0 + u, 1.5, 2.0 - 2 * u, 2.0 - u], rng.uniform(1.0, 2.0, 59)])
    return np.ldexp(m[None, :], np.arange(lo, hi + 1)[:, None]).ravel()


def off(got, want):
    """Largest error in units of 2^-53 of the value."""
    return float(np.abs((got.astype(np.longdouble) - want) / want).max() * np.longdouble(2.0) ** 53)


def test_long_doubles_have_64_bits():
    assert np.finfo(np.longdouble).nmant >= 63


def test_reciprocal():
    x = every_exponent(-1022, 1020, 0)          # 1/x normal too
    assert off(device(RCP, x), 1 / x.astype(np.longdouble)) <= 1.01
    # where 1/x is below the normal range it may be 0
    x = every_exponent(1021, 1023, 1)
    got = device(RCP, x)
    assert (np.abs(got - 1.0 / x) <= 2.0 ** -1022).all()


def test_reciprocal_square_root():
    x = every_exponent(-1022, 1023, 2)
    assert off(device(RSQRT, x), 1 / np.sqrt(x.astype(np.longdouble))) <= 1.6


def test_exponential():
    rng = np.random.default_rng(3)
    k = np.arange(-32672.0, 1.0)                # every table entry at every exponent, and between two
    y = np.concatenate([k, k[1:] - 0.5, np.nextafter(k[1:] - 0.5, 0.0), np.nextafter(k[1:] - 0.5, -1e9),
                        rng.uniform(-32672.0, 0.0, 200000), rng.uniform(-64.0, 0.0, 200000),
                        -np.ldexp(rng.uniform(1.0, 2.0, 4000), rng.integers(-1022, 0, 4000))])
    assert y.min() == -32672.0 and y.max() == 0.0
    assert off(device(EXP, y), np.exp2(y.astype(np.longdouble) / 32)) <= 2.1
