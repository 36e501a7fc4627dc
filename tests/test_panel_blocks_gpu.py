"""The blocked Gauss-Jordan inverse of the panel system (csrc/vx_gj.cu) at
the sizes where its blocks end: steps in blocks of 16 (P a multiple of 16, one
more, one less), rows 512 to a thread block of the panel cluster (P + 1 = 512
and 513, three blocks at 1030), strips of 8 columns.  Against the oracle's
column-by-column elimination (the reference's rule), within the 1e-11 of the
largest entry that the device matrix of a circle is held to at 200 and 1000
panels; with partial pivoting, an inverse of the oracle's influence matrix as
good as that: |M L - 1| within 1e-11 (P + 1) max |M| max |L|."""
import ctypes as C

import numpy as np
import pytest

from oracle import oracle as O
from vortex_b200 import native as N
from vortex_b200 import profiles

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("P", [15, 16, 17, 33, 511, 512, 1030])
def test_blocked_inverse(P):
    pan = profiles.ellipse(P, 0.5, 0.4)
    L, M = np.zeros((P + 1, P + 1)), np.zeros((P + 1, P + 1))
    assert O.lib().vxo_panel_matrix(C.c_void_p(pan.ctypes.data), C.c_int64(P), C.c_void_p(L.ctypes.data),
                                    C.c_void_p(M.ctypes.data)) == 0
    got = {}
    for mode in (0, 1):
        sim = N.Sim(N.default_conf(ve_size=float(pan["length"].mean()), gj_pivot=mode), pan)
        got[mode] = sim.matrix()
        sim.close()
    assert np.abs(got[0] - M).max() <= 1e-11 * np.abs(M).max()
    assert np.abs(got[1] @ L - np.eye(P + 1)).max() <= 1e-11 * (P + 1) * np.abs(got[1]).max() * np.abs(L).max()
