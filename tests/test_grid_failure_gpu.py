"""A diffusion grid that cannot be made (a vortex whose position is a NaN
with its sign set, infinite, or beyond all range): the stage reports it,
orders nothing and leaves the body's vortices and everything else on the
device as they were, on a body's first grid as after good ones, in one call
with the velocity, by itself and in a whole step; a body beside it goes on
with the same bits."""
import numpy as np
import pytest

from tests.helpers import conf_kwargs, wake_cloud
from vortex_b200 import native as N
from vortex_b200 import profiles

pytestmark = pytest.mark.gpu


def body(x, y, g):
    sim = N.Sim(N.default_conf(**conf_kwargs(200, precision=N.PREC_FP32)), profiles.circle(200))
    sim.set_particles(x, y, g)
    return sim


@pytest.mark.parametrize("n", [2, 33, 5000])
@pytest.mark.parametrize("bad", ["nan_x", "nan_y", "nan_xy", "inf_x", "inf_xy", "far_xy"])
def test_grid_that_cannot_be_made(n, bad):
    x, y, g = wake_cloud(n, seed=n)
    good = (x, y, g)
    value = {"nan": -np.nan, "inf": np.inf, "far": 1e60}[bad[:3]]
    bx, by = x.copy(), y.copy()
    if "x" in bad[4:]:
        bx[n // 2] = value
    if "y" in bad[4:]:
        by[n // 2] = value
    beside, alone = body(*good), body(*good)
    for calls in ([("velocity", "diffusion")], [("velocity",), ("diffusion",)], "step"):
        for first in (True, False):
            sim = body(*good)
            if not first:
                sim.stage("velocity", "diffusion")
            sim.set_particles(bx, by, g)
            if calls == "step":
                sim.step(1)
                with pytest.raises(N.VxError):
                    sim.count()
            else:
                if len(calls) == 2:
                    sim.stage(*calls[0])
                with pytest.raises(N.VxError):
                    sim.stage(*calls[-1])
                for got, set_ in zip(sim.get_slots(n), (bx, by, g)):
                    assert np.array_equal(got, set_, equal_nan=True)
            beside.stage("velocity", "diffusion")
            sim.close()
    alone.stage("velocity", "diffusion")
    for a, b in zip(beside.velocity(), alone.velocity()):
        assert np.array_equal(a, b)
    beside.close()
    alone.close()
