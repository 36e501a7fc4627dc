"""The blocked Gauss-Jordan inverse (csrc/vx_gj.cu) against the column-by-column
elimination it reorders, bit for bit, where its cluster changes: one thread
block takes up to 128 matrix rows, a further one each further 128 up to eight,
which take up to 512 rows each beyond; the largest system the cluster takes is
that of 4095 panels, and one of 4096 goes column by column in either call.
Both pivot rules, an ellipse and the rounded plate."""
import ctypes as C

import numpy as np
import pytest

from vortex_b200 import native as N
from vortex_b200 import profiles

pytestmark = pytest.mark.gpu


def inverse(pan, robust, columns):
    P = len(pan)
    M = np.zeros((P + 1, P + 1))
    status = N.lib().vx_eval_inverse(C.c_void_p(pan.ctypes.data), C.c_int64(P), C.c_int(robust), C.c_int(columns),
                                     C.c_void_p(M.ctypes.data))
    return status, M


@pytest.mark.parametrize("shape", ["ellipse", "plate"])
@pytest.mark.parametrize("P", [16, 126, 127, 128, 129, 254, 255, 895, 896, 1022, 1023, 1024, 2100])
def test_blocks_and_columns(P, shape):
    pan = profiles.ellipse(P, 0.5, 0.3) if shape == "ellipse" else profiles.rotate(profiles.rounded_plate(P), -20.0)
    for robust in (0, 1):
        (sa, a), (sb, b) = inverse(pan, robust, 0), inverse(pan, robust, 1)
        assert sa == sb
        if shape == "ellipse" or robust:    # the reference's rule may meet a pivot below its threshold
            assert sa == 0
        if sa == 0:
            assert np.isfinite(b).all() and np.array_equal(a, b)


@pytest.mark.parametrize("P", [4095, 4096])
def test_largest_system(P):
    pan = profiles.circle(P)
    (sa, a), (sb, b) = inverse(pan, 0, 0), inverse(pan, 0, 1)
    assert sa == sb == 0 and np.isfinite(a).all() and np.array_equal(a, b)
