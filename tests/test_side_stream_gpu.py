"""The bulk form's second stream (the 3 nearest and the diffusion grid beside
the expansions and the near field): a step, the two stages in one call, and
several bodies stepped in turn give the bits of the same work one launch
after the other (timed kernels, one stage a call), from one vortex to enough
to fill the GPU; a body grown and reset between steps; two bodies at once."""
import numpy as np
import pytest

from tests.helpers import conf_kwargs, wake_cloud
from vortex_b200 import native as N
from vortex_b200 import profiles

pytestmark = pytest.mark.gpu


def body(n, seed=0):
    sim = N.Sim(N.default_conf(**conf_kwargs(200, precision=N.PREC_FP32)), profiles.circle(200))
    sim.set_particles(*wake_cloud(n, seed=seed))
    return sim


def state(sim):
    return [np.array(a) for a in sim.particles()] + [np.array(a) for a in sim.velocity()]


def same(a, b):
    assert all(np.array_equal(p, q) for p, q in zip(a, b))


@pytest.mark.parametrize("n", [1, 33, 1000, 20000, 300000])
def test_step_beside_and_in_turn(n):
    a, b, c = body(n), body(n), body(n)
    a.step(4)
    b.kernel_times(4)               # every launch timed: one after the other
    for _ in range(4):              # two bodies' steps on the device at once
        c.step(1)
        a2 = body(n, seed=1)
        a2.step(2)
        a2.close()
    same(state(a), state(b))
    same(state(a), state(c))
    a.set_particles(*wake_cloud(2 * n, seed=2))     # grows
    b.set_particles(*wake_cloud(2 * n, seed=2))
    a.step(2)
    b.kernel_times(2)
    same(state(a), state(b))
    for s in (a, b, c):
        s.close()


@pytest.mark.parametrize("n", [1, 700, 40000])
def test_stages_in_one_call(n):
    a, b = body(n), body(n)
    for _ in range(3):
        a.stage("velocity", "diffusion")
        b.stage("velocity")
        b.stage("diffusion")
        same(state(a), state(b))
    a.close()
    b.close()


def test_batch_of_all_forms():
    """Bodies whose steps have two branches, one branch (direct sums) and the
    plain form in one batch: each as stepped alone."""
    kinds = [dict(precision=N.PREC_FP32), dict(precision=N.PREC_FP32, fmm=0), dict(precision=N.PREC_FP64),
             dict(precision=N.PREC_FP32, fmm_p=8), dict(precision=N.PREC_FP32, diff_cutoff=0.0, fmm=0)]

    def build():
        out = []
        for k, kw in enumerate(kinds * 2):
            sim = N.Sim(N.default_conf(**conf_kwargs(60 + 40 * k, **kw)), profiles.circle(60 + 40 * k))
            sim.set_particles(*wake_cloud(300 + 700 * k, seed=k))
            out.append(sim)
        return out

    alone, members = build(), build()
    batch = N.Batch(members)
    for steps in (1, 4):
        batch.step(steps)
        for s in alone:
            s.step(steps)
    batch.close()
    for a, m in zip(alone, members):
        same(state(a), state(m))
        a.close()
        m.close()
