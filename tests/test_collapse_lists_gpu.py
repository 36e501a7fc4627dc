"""Candidate lists of the collapse's settling block at the sizes where its
rounds change (one candidate a thread, up to 1024; four at a time beyond):
groups of two, three or five vortices closer than the merge radius, far from
the other groups, in a random order, so that candidates share partners, take
one another and wait for one another.  Against the oracle, every slot bit for
bit, over two passes."""
import numpy as np
import pytest

from oracle import oracle as O
from tests.helpers import conf_kwargs, oracle_params, with_tail
from vortex_b200 import native as N
from vortex_b200 import profiles

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_col", [1, 2])
@pytest.mark.parametrize("pas", [1, 2])
@pytest.mark.parametrize("size", [2, 3, 5])
@pytest.mark.parametrize("groups", [1023, 1024, 1025, 4096, 4097])
def test_candidate_lists(groups, size, pas, n_col):
    rng = np.random.default_rng(groups + size)
    n = groups * size
    k = rng.permutation(np.repeat(np.arange(groups), size))
    x = 0.6 + 0.1 * (k % 65) + rng.uniform(-1e-3, 1e-3, n)
    y = -3.2 + 0.1 * (k // 65) + rng.uniform(-1e-3, 1e-3, n)
    g = rng.choice([1e-3, 2e-3], n) * (rng.choice([-1.0, 1.0], n) if pas == 1 else 1.0)
    ck = conf_kwargs(200, r_col_diff_sign=0.3, r_col_same_sign=0.3, max_ve_g=6e-3, n_col=n_col)
    pan = profiles.circle(200)
    sim = N.Sim(N.default_conf(**ck), pan)
    p = oracle_params(pan, ck)
    xs, ys, gs = with_tail(x, y, g, extra=32)
    sim.set_slots(xs, ys, gs, n)
    for _ in range(2):
        sim.stage("collapse1" if pas == 1 else "collapse2")
        before = n
        xs, ys, gs, n = O.collapse(p, pas, xs, ys, gs, n)
        assert sim.count() == n
        for got, want in zip(sim.get_slots(len(xs)), (xs, ys, gs)):
            assert np.array_equal(got, want)
        assert _ == 1 or before - n >= groups // 4
    sim.close()
