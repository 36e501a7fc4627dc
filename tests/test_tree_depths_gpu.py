"""The quadtree's passes at every depth a small body has: clouds that give
trees of depth 2 (the box rule's least) to 6, quadtree levels of which the
upward pass sums two in its first kernel, none or some in its second, with
full and nearly empty leaves, for each expansion order.  Bulk velocity against
the plain FP64 sums: within 2e-5 of the largest (the bulk form's stated bound);
order 8 within 1e-3, its truncation (0.55^9 of a source's far field)."""
import numpy as np
import pytest

from tests.helpers import conf_kwargs, wake_cloud
from vortex_b200 import native as N
from vortex_b200 import profiles

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,depth", [(33, 2), (600, 3), (3000, 4), (9000, 5), (40000, 6)])
def test_bulk_velocity_by_depth(n, depth):
    pan = profiles.circle(200)
    x, y, g = wake_cloud(n, seed=n)
    ck = conf_kwargs(200)
    plain = N.Sim(N.default_conf(**dict(ck, precision=N.PREC_FP64)), pan)
    plain.set_particles(x, y, g)
    plain.stage("velocity")
    u, v, _ = plain.velocity()
    plain.close()
    scale = np.hypot(u, v).max()
    for order in (8, 12, 16, 20):
        sim = N.Sim(N.default_conf(**dict(ck, precision=N.PREC_FP32, fmm_p=order)), pan)
        sim.set_particles(x, y, g)
        sim.stage("velocity")
        a, b, _ = sim.velocity()
        assert sim.tree_info()["fmm_level"] == depth
        sim.close()
        assert np.hypot(a - u, b - v).max() <= (1e-3 if order == 8 else 2e-5) * scale, order
