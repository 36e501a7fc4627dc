"""A bulk body made with the direct sums and switched to the quadtree later (as
the autotuner does), back and again, computes what one made with it does, bit for
bit: stages in one call, steps, in a batch."""
import numpy as np
import pytest

from tests.helpers import conf_kwargs, wake_cloud
from vortex_b200 import native as N
from vortex_b200 import profiles

pytestmark = pytest.mark.gpu


def body(n, fmm, **kw):
    sim = N.Sim(N.default_conf(**conf_kwargs(200, **{**dict(precision=N.PREC_FP32, fmm=fmm), **kw})), profiles.circle(200))
    sim.set_particles(*wake_cloud(n, seed=n))
    return sim


def same(a, b):
    assert all(np.array_equal(p, q) for p, q in zip([*a.particles(), *a.velocity()], [*b.particles(), *b.velocity()]))


@pytest.mark.parametrize("n", [1, 700, 40000])
def test_switched_later(n):
    made, switched = body(n, 1), body(n, 0)
    for _ in range(2):
        switched.set_fmm(False, 32)
        switched.set_fmm(True, 32)
        for sim in (made, switched):
            sim.stage("velocity", "diffusion")
        same(made, switched)
        for sim in (made, switched):
            sim.step(2)
        same(made, switched)
    batch = N.Batch([switched])
    batch.step(2)
    made.step(2)
    batch.close()
    same(made, switched)
    made.close()
    switched.close()


def test_plain_body_takes_the_switch():
    a, b = body(700, 0, precision=N.PREC_FP64), body(700, 1, precision=N.PREC_FP64)
    a.set_fmm(True, 32)
    for sim in (a, b):
        sim.step(2)
    same(a, b)
    a.close()
    b.close()
