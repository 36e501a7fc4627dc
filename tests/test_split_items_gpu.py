"""The bulk diffusion where its work is split over more warps (csrc/vx_cells.cu:
8, 4, 2 or 1 warps an item by the body's item count, 8, 2 or 1 a wide target)
and the 3-nearest search over squares of leaves (csrc/vx_fmm.cu), on Gaussian
clouds whose edges are sparse, with a few vortices far out (a window of many
rows, the widest square, the scan of every source).  Strengths of one sign, so
that no sum cancels: distance within 2e-6 of the plain form's, diffusion
increment within 1e-4 of the largest (the bounds test_edges_gpu holds)."""
import numpy as np
import pytest

from tests.helpers import conf_kwargs
from vortex_b200 import native as N
from vortex_b200 import profiles

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [40, 1000, 9000, 20000, 40000, 70000])
def test_split_diffusion_and_squares(n):
    rng = np.random.default_rng(n)
    x, y = rng.normal(3.0, 0.5, n), rng.normal(0.0, 0.25, n)
    far = max(1, n // 2000)
    x[:far] += rng.uniform(2.0, 6.0, far)
    y[:far] += rng.uniform(-8.0, 8.0, far)
    g = rng.uniform(1e-4, 1e-3, n)
    ck = conf_kwargs(200)
    got = {}
    d = None
    for form in (N.PREC_FP64, N.PREC_FP32):
        sim = N.Sim(N.default_conf(**dict(ck, precision=form)), profiles.circle(200))
        sim.set_particles(x, y, g)
        sim.stage("velocity")
        u, v, dist = sim.velocity()
        if d is None:
            d = dist
        else:
            assert np.abs(dist - d).max() <= 2e-6 * d.max()
        sim.set_velocity(np.zeros(n), np.zeros(n), d)
        sim.stage("diffusion")
        got[form] = sim.velocity()[:2]
        sim.close()
    (a, b), (p, q) = got[N.PREC_FP64], got[N.PREC_FP32]
    scale = np.hypot(a, b).max()
    assert np.hypot(a - p, b - q).max() <= 1e-4 * scale
