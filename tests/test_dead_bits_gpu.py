"""Compaction from the bitmap of dead vortices (csrc/vx_compact.cuh) against the
oracle, every slot bit for bit: counts at the edges of a bitmap word, of a
16-byte load and of a block's round, none, few, half or all of them dead, the
first or the last, NaN strengths, more than the marking kernel's last block
removes by itself, the same state compacted twice; and the same inside a
collapse that starts from a state with vortices too weak to stay."""
import numpy as np
import pytest

from oracle import oracle as O
from tests.helpers import conf_kwargs, oracle_params, with_tail
from vortex_b200 import native as N
from vortex_b200 import profiles

pytestmark = pytest.mark.gpu


def same(sim, xs, ys, gs, n):
    assert sim.count() == n
    gx, gy, gg = sim.get_slots(len(xs))
    assert np.array_equal(gx, xs) and np.array_equal(gy, ys) and np.array_equal(gg, gs)


@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 127, 128, 129, 1000, 4095, 4096, 4097, 40000, 131200])
@pytest.mark.parametrize("dead", ["none", "first", "last", "few", "half", "all", "nan"])
def test_compact_bits(n, dead):
    rng = np.random.default_rng(n)
    x, y, g = rng.normal(2, 1, n), rng.normal(0, 1, n), rng.choice([-1e-3, 2e-3], n)
    kill = {"none": [], "first": [0], "last": [n - 1], "all": np.arange(n),
            "few": rng.integers(0, n, 1 + n // 500), "nan": rng.integers(0, n, 1 + n // 300),
            "half": np.flatnonzero(rng.random(n) < 0.5)}[dead]
    g[kill] = np.nan if dead == "nan" else 1e-13
    sim = N.Sim(N.default_conf(**conf_kwargs(200)), profiles.circle(200))
    xs, ys, gs = with_tail(x, y, g, extra=32)
    sim.set_slots(xs, ys, gs, n)
    for _ in range(2):
        sim.stage("compact")
        if dead == "nan":   # the oracle's serial loop keeps to the same rule with a weak strength
            gs = np.where(np.isnan(gs), 1e-13, gs)
        xs, ys, gs, n = O.compact(xs, ys, gs, n)
        same(sim, xs, ys, gs, n)
    sim.close()


@pytest.mark.parametrize("n_col", [1, 2, 3])
@pytest.mark.parametrize("pas", [1, 2])
def test_collapse_of_weak(pas, n_col):
    rng = np.random.default_rng(pas)
    n, groups = 6000, 500
    cx, cy, k = rng.uniform(0.6, 3.0, groups), rng.normal(0, 0.4, groups), rng.integers(0, groups, n)
    x, y = cx[k] + rng.normal(0, 0.003, n), cy[k] + rng.normal(0, 0.003, n)
    g = rng.choice([1e-3, 2e-3, -1e-3], n)
    g[rng.random(n) < 0.3] *= 1e-10     # weak, not zero: they may merge in the first round
    ck = conf_kwargs(200, r_col_diff_sign=0.3, r_col_same_sign=0.25, max_ve_g=6e-3, n_col=n_col)
    pan = profiles.circle(200)
    sim = N.Sim(N.default_conf(**ck), pan)
    p = oracle_params(pan, ck)
    xs, ys, gs = with_tail(x, y, g, extra=32)
    sim.set_slots(xs, ys, gs, n)
    for _ in range(2):
        sim.stage("collapse1" if pas == 1 else "collapse2")
        xs, ys, gs, n = O.collapse(p, pas, xs, ys, gs, n)
        same(sim, xs, ys, gs, n)
    sim.close()


@pytest.mark.parametrize("n_col", [1, 2, 3])
@pytest.mark.parametrize("pas", [1, 2])
def test_collapse_of_many(pas, n_col):
    """In a store of more than 65536 slots a round with more than 1024 dead
    leaves the moves to further launches, the second round's renaming too."""
    rng = np.random.default_rng(7 + pas)
    n, groups = 20000, 1500
    cx, cy, k = rng.uniform(0.6, 3.0, groups), rng.normal(0, 0.4, groups), rng.integers(0, groups, n)
    x, y = cx[k] + rng.normal(0, 0.004, n), cy[k] + rng.normal(0, 0.004, n)
    g = rng.choice([1e-3, 2e-3, -1e-3], n)
    ck = conf_kwargs(200, r_col_diff_sign=0.3, r_col_same_sign=0.25, max_ve_g=6e-3, n_col=n_col)
    pan = profiles.circle(200)
    sim = N.Sim(N.default_conf(**ck), pan)
    p = oracle_params(pan, ck)
    sim.set_particles(rng.uniform(1, 3, 70001), rng.uniform(-1, 1, 70001), np.full(70001, 1e-3))
    xs, ys, gs = with_tail(x, y, g, extra=32)
    sim.set_slots(xs, ys, gs, n)
    for _ in range(2):
        sim.stage("collapse1" if pas == 1 else "collapse2")
        before = n
        xs, ys, gs, n = O.collapse(p, pas, xs, ys, gs, n)
        same(sim, xs, ys, gs, n)
        assert _ == 1 or before - n > 2048
    sim.close()
