"""The collapse's second round on the first one's grid (csrc/vx_collapse.cu)
against the oracle's rounds, every slot bit for bit: chains of merges whose
results merge again, vortices the compaction moves into holes, merged ones
that are dropped (opposite signs that cancel), a box so wide that the cells
grow beyond the merge radius, one and two vortices, none that merges; one,
two and four rounds, and a second collapse right after the first (its
arrays must be clear)."""
import numpy as np
import pytest

from oracle import oracle as O
from tests.helpers import conf_kwargs, oracle_params, with_tail
from vortex_b200 import native as N
from vortex_b200 import profiles

pytestmark = pytest.mark.gpu


def scene(kind, rng):
    if kind == "few":
        return np.array([1.0, 1.001]), np.array([0.0, 0.0]), np.array([1e-3, 2e-3])
    if kind == "apart":
        x, y = np.meshgrid(np.arange(40) * 0.1 + 1.0, np.arange(30) * 0.1 - 1.5)
        return x.ravel(), y.ravel(), rng.normal(0, 1e-3, 1200)
    n, groups = (20000, 1500) if kind == "dense" else (4000, 300)
    cx, cy = rng.uniform(0.6, 3.0, groups), rng.normal(0, 0.4, groups)
    k = rng.integers(0, groups, n)
    x, y = cx[k] + rng.normal(0, 0.004, n), cy[k] + rng.normal(0, 0.004, n)
    g = rng.choice([1e-3, 2e-3, -1e-3], n)      # opposite ones cancel exactly
    if kind == "wide":
        x[:20] += rng.uniform(-1.5, 6.0, 20)
        y[:20] += rng.uniform(-9.0, 9.0, 20)
    return x, y, g


@pytest.mark.parametrize("n_col", [1, 2, 4])
@pytest.mark.parametrize("pas", [1, 2])
@pytest.mark.parametrize("kind", ["few", "apart", "chains", "wide", "dense"])
def test_collapse_rounds(kind, pas, n_col):
    rng = np.random.default_rng(len(kind) + pas)
    x, y, g = scene(kind, rng)
    n = len(x)
    ck = conf_kwargs(200, r_col_diff_sign=0.3, r_col_same_sign=0.25, max_ve_g=6e-3, n_col=n_col)
    if kind == "wide":
        ck["ve_size"] = 0.004
        ck["r_col_diff_sign"], ck["r_col_same_sign"] = 0.5, 0.4
    pan = profiles.circle(200)
    sim = N.Sim(N.default_conf(**ck), pan)
    p = oracle_params(pan, ck)
    xs, ys, gs = with_tail(x, y, g, extra=32)
    sim.set_slots(xs, ys, gs, n)
    for _ in range(2):
        sim.stage("collapse1" if pas == 1 else "collapse2")
        xs, ys, gs, n = O.collapse(p, pas, xs, ys, gs, n)
        assert sim.count() == n
        gx, gy, gg = sim.get_slots(len(xs))
        assert np.array_equal(gx, xs) and np.array_equal(gy, ys) and np.array_equal(gg, gs)
    sim.close()
