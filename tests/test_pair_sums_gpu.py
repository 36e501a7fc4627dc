"""The plain form's pair sums (csrc/vx_pairs.cu) where their tiles and source
chunks end, and where a pair is at its limits: one warp, one tile of 512
targets more or less one, enough vortices for several chunks; coincident
vortices, a vortex 1e7 away (its exponential underflows), one at an infinite
squared distance (1e200).  Against the same sums in numpy: the 3-nearest
distance to the last bit, velocities within 1e-12 of the largest (sum order
and a last bit of each term, as test_parity_gpu holds them)."""
import math

import numpy as np
import pytest

from tests.helpers import conf_kwargs
from vortex_b200 import native as N
from vortex_b200 import profiles

pytestmark = pytest.mark.gpu


def numpy_sums(x, y, g, eps, nu):
    n = len(x)
    u, v, d, du, dv = (np.zeros(n) for _ in range(5))
    with np.errstate(over="ignore", invalid="ignore", divide="ignore"):
        for i in range(n):
            dx, dy = x[i] - x, y[i] - y
            r2 = dx * dx + dy * dy
            w = g / np.maximum(r2, eps * eps)
            u[i] = -np.sum(w * dy) / (2 * math.pi) + 1.0
            v[i] = np.sum(w * dx) / (2 * math.pi)
            r = np.sqrt(r2)
            d[i] = np.minimum(np.sort(np.delete(r, i))[:3], math.sqrt(1e5)).sum() / 3
            far = r > 0.001 * eps
            e = np.where(far, g * np.exp(-r / d[i]), 0.0)
            i1 = e.sum()
            if abs(i1) > 1e-5:
                m = np.where(far & np.isfinite(r), e / np.where(far, r, 1.0), 0.0)
                du[i], dv[i] = nu * np.sum(m * dx) / (i1 * d[i]), nu * np.sum(m * dy) / (i1 * d[i])
    return u, v, d, u + du, v + dv


@pytest.mark.parametrize("n", [1, 2, 33, 511, 512, 513, 2049])
@pytest.mark.parametrize("odd", ["none", "coincident", "far", "infinite"])
def test_plain_pair_sums(n, odd):
    rng = np.random.default_rng(n)
    x, y, g = rng.uniform(1.0, 3.0, n), rng.uniform(-1.0, 1.0, n), rng.uniform(1e-4, 2e-4, n)
    if odd == "coincident":
        x[: n // 2], y[: n // 2] = x[0], y[0]
    elif odd == "far":
        x[-1] = 1e7
    elif odd == "infinite":
        x[-1] = 1e200
    ck = conf_kwargs(200)
    sim = N.Sim(N.default_conf(**dict(ck, precision=N.PREC_FP64)), profiles.circle(200))
    sim.set_particles(x, y, g)
    sim.stage("velocity")
    u, v, d = sim.velocity()
    ru, rv, rd, su, sv = numpy_sums(x, y, g, ck["ve_size"], ck["viscosity"])
    near = slice(0, n - 1) if odd in ("far", "infinite") else slice(0, n)   # the far vortex: d is the padding's
    scale = np.hypot(ru, rv).max()
    assert np.abs(u - ru).max() <= 1e-12 * scale and np.abs(v - rv).max() <= 1e-12 * scale
    if n > 4:
        assert np.abs(d - rd)[near].max() <= 4 * np.spacing(rd[near].max())
        sim.set_velocity(d=rd)
        sim.stage("diffusion")
        a, b, _ = sim.velocity()
        scale = np.hypot(su, sv)[near].max()
        assert np.abs(a - su)[near].max() <= 1e-12 * scale and np.abs(b - sv)[near].max() <= 1e-12 * scale
    sim.close()


@pytest.mark.parametrize("points", [1, 33, 511, 512, 513, 1024, 1025, 5000])
@pytest.mark.parametrize("n", [1, 300, 20000])
def test_probe_points(points, n):
    """Probe velocities at the sizes where the tiles and the two-target form
    end: plain form against the sums in numpy within 1e-12 of the largest, bulk
    form within 2e-5 of it (the bulk form's stated velocity bound)."""
    rng = np.random.default_rng(points + n)
    x, y, g = rng.uniform(1.0, 3.0, n), rng.uniform(-1.0, 1.0, n), rng.normal(0.0, 1e-3, n)
    px, py = rng.uniform(0.0, 4.0, points), rng.uniform(-2.0, 2.0, points)
    ck = conf_kwargs(200)
    ref = np.zeros((2, points))
    for a in range(0, points, 500):
        dx, dy = px[a:a + 500, None] - x, py[a:a + 500, None] - y
        w = g / np.maximum(dx * dx + dy * dy, ck["ve_size"] ** 2)
        ref[:, a:a + 500] = 1.0 - (w * dy).sum(1) / (2 * math.pi), (w * dx).sum(1) / (2 * math.pi)
    scale = np.abs(ref).max()
    for form, tol in ((N.PREC_FP64, 1e-12), (N.PREC_FP32, 2e-5)):
        sim = N.Sim(N.default_conf(**dict(ck, precision=form)), profiles.circle(200))
        sim.set_particles(x, y, g)
        u, v = sim.probe(px, py)
        sim.close()
        assert np.abs(u - ref[0]).max() <= tol * scale and np.abs(v - ref[1]).max() <= tol * scale
