"""The bulk form's all-pairs diffusion (no cut-off) takes the vortices as they
are, whichever stage or call came before it: after the quadtree's velocity and
after the direct sums', by itself, in one call, in a whole step, alone and in
a batch, when the last packed sources were those of another cloud.

The stage by itself against the plain form's on the same distances d.
Vortices on a jittered grid lie at least 0.01 apart at coordinates below 4: a
rounded coordinate difference is off by up to 2.4e-7, a term of the sums (of
one sign) by up to 2.4e-5 of itself in direction, 6e-6 in its exponential at
d = 0.04 and a few 1e-6 in the approximations, so a diffusive velocity nu I2 /
(I1 d) by less than 1e-4 nu / d."""
import numpy as np
import pytest

from tests.helpers import conf_kwargs, wake_cloud
from vortex_b200 import native as N
from vortex_b200 import profiles

pytestmark = pytest.mark.gpu


def cloud(n, seed):
    rng = np.random.default_rng(seed)
    k = rng.choice(40 * 80, n, replace=False)
    return (1.0 + 0.05 * (k % 40 + rng.uniform(0.1, 0.9, n)), -2.0 + 0.05 * (k // 40 + rng.uniform(0.1, 0.9, n)),
            rng.uniform(1e-4, 2e-4, n))


def body(n, fmm, seed=0, **kw):
    """A body whose last packed sources are another cloud's."""
    ck = conf_kwargs(200, **{**dict(precision=N.PREC_FP32, diff_cutoff=0.0, fmm=fmm), **kw})
    sim = N.Sim(N.default_conf(**ck), profiles.circle(200))
    sim.set_particles(*wake_cloud(n, seed=99))
    sim.probe([2.0], [0.0])
    sim.set_particles(*cloud(n, seed))
    return sim


def state(sim):
    return [np.array(a) for a in sim.particles()] + [np.array(a) for a in sim.velocity()]


def same(a, b):
    assert all(np.array_equal(p, q) for p, q in zip(a, b))


@pytest.mark.parametrize("fmm", [0, 1])
@pytest.mark.parametrize("n", [33, 1025, 3000])
def test_stage_by_itself(n, fmm):
    plain, bulk = body(n, 0, precision=N.PREC_FP64), body(n, fmm)
    plain.stage("velocity")
    d = plain.velocity()[2]
    for sim in (plain, bulk):
        sim.set_velocity(vx=np.zeros(n), vy=np.zeros(n), d=d)
        sim.stage("diffusion")
    nu = conf_kwargs(200)["viscosity"]
    for a, b in zip(bulk.velocity()[:2], plain.velocity()[:2]):
        assert (np.abs(a - b) <= 1e-4 * nu / d).all()
    plain.close()
    bulk.close()


@pytest.mark.parametrize("fmm", [0, 1])
@pytest.mark.parametrize("n", [33, 1025, 3000])
def test_calls_agree(n, fmm):
    a, b, c, m = (body(n, fmm) for _ in range(4))
    batch = N.Batch([m])
    for _ in range(2):
        a.stage("velocity", "diffusion", "wall")
        b.stage("velocity")
        b.stage("diffusion")
        b.stage("wall")
        same(state(a), state(b))
    a.set_particles(*cloud(n, 1))
    b.set_particles(*cloud(n, 1))
    c.set_particles(*cloud(n, 1))
    batch.remove(m)
    m.set_particles(*cloud(n, 1))
    batch.add(m)
    for _ in range(2):
        a.step(1)
        b.kernel_times(1)
        batch.step(1)
        for st in ("birth", "velocity", "diffusion", "wall", "advect", "compact", "collapse1", "collapse2"):
            c.stage(st)
        same(state(a), state(b))
        same(state(a), state(c))
        same(state(a), state(m))
    batch.close()
    for s in (a, b, c, m):
        s.close()
