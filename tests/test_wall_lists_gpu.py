"""The wall term where its work lists end (csrc/vx_wall.cu): particles in
groups of 32 an eighth of the array apart, lists of up to 256 a block, panels
32 at a time: one particle, one group more or less one, every particle near
the wall or one in a hundred, and a small fine body whose cells list more
panels than a warp has lanes (a thin plate, both sides).  Plain form
against the oracle within 1e-13 of velocities of order 1 (as
test_parity_gpu); bulk form within 2e-5 of the plain one, the bulk form's
stated bound."""
import numpy as np
import pytest

from oracle import oracle as O
from tests.helpers import conf_kwargs, oracle_params
from vortex_b200 import native as N
from vortex_b200 import profiles

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", ["circle", "plate"])
@pytest.mark.parametrize("n,near", [(1, 1.0), (31, 1.0), (33, 1.0), (257, 1.0), (2500, 1.0), (20000, 0.01)])
def test_wall_lists(shape, n, near):
    pan = profiles.circle(200) if shape == "circle" else profiles.rounded_plate(400)
    rng = np.random.default_rng(n)
    k = rng.integers(0, len(pan), n)
    off = pan["length"][k] * rng.uniform(0.2, 6.0, n)
    off[: n // 10] = 1.00001e-4        # within a tenth of a panel of a birth point
    x = pan["left"][k, 0] + off * pan["norm"][k, 0]
    y = pan["left"][k, 1] + off * pan["norm"][k, 1]
    away = rng.random(n) > near
    x[away] += 3.0
    d = rng.uniform(0.5, 3.0, n) * pan["length"].mean()
    ck = conf_kwargs(len(pan), ve_size=float(pan["length"].mean()))
    got = {}
    for form in (N.PREC_FP64, N.PREC_FP32):
        sim = N.Sim(N.default_conf(**dict(ck, precision=form, gj_pivot=2)), pan)
        sim.set_particles(x, y, np.full(n, 1e-3))
        sim.set_velocity(np.ones(n), np.zeros(n), d)
        sim.stage("wall")
        got[form] = sim.velocity()[:2]
        sim.close()
    ex, ey = O.wall_diffusion(oracle_params(pan, ck), pan, x, y, n, d, np.ones(n), np.zeros(n))
    scale = max(1.0, np.abs(ex).max(), np.abs(ey).max())
    u, v = got[N.PREC_FP64]
    assert np.abs(u - ex).max() < 1e-13 * scale and np.abs(v - ey).max() < 1e-13 * scale
    a, b = got[N.PREC_FP32]
    assert np.abs(a - u).max() <= 2e-5 * scale and np.abs(b - v).max() <= 2e-5 * scale
