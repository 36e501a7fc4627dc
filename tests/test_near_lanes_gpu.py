"""Work dealt out within a warp in the quadtree's near field and 3-nearest
search (csrc/vx_fmm.cu): clusters of 1 to 70 vortices far apart, so that a
leaf's last item holds any number of targets (a whole, half or quarter warp to
each) and a target's three neighbours lie in its own quarter leaf, across an
edge, a corner or two leaves away; pairs, triples and a single vortex.  Bulk
form against the plain FP64 form: velocity within 2e-5 of the largest,
distance within 2e-6 of the largest (the bounds test_tree_depths_gpu and
test_split_items_gpu hold)."""
import numpy as np
import pytest

from tests.helpers import conf_kwargs
from vortex_b200 import native as N
from vortex_b200 import profiles

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [[1], [2], [3], [5, 4], [7, 8, 9], [15, 16, 17, 18], [31, 32, 33],
                                   list(range(1, 71)), list(range(70, 0, -1)) * 4])
def test_clusters(sizes):
    rng = np.random.default_rng(len(sizes))
    xs, ys = [], []
    for q, k in enumerate(sizes):
        xs.append(0.8 + 0.21 * (q % 20) + rng.uniform(0.0, 0.08, k))
        ys.append(-1.5 + 0.23 * (q // 20) + rng.uniform(0.0, 0.08, k))
    x, y = np.concatenate(xs), np.concatenate(ys)
    g = rng.uniform(1e-3, 2e-3, len(x))
    got = []
    for form in (N.PREC_FP64, N.PREC_FP32):
        sim = N.Sim(N.default_conf(**conf_kwargs(200, precision=form)), profiles.circle(200))
        sim.set_particles(x, y, g)
        sim.stage("velocity")
        got.append(sim.velocity())
        sim.close()
    (u, v, d), (a, b, c) = got
    assert np.hypot(a - u, b - v).max() <= 2e-5 * np.hypot(u, v).max()
    assert np.abs(c - d).max() <= 2e-6 * d.max()
