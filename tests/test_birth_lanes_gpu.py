"""The bulk birth's near panel terms with 8, 4 or 1 lanes a panel
(csrc/vx_birth.cu) at counts around a staged tile of 128 sources, a chunk
and a group of 8, for panel counts around a block's panels: born strengths
within 1e-5 of the largest of the plain FP64 form's (the bound test_bulk_gpu
holds)."""
import math

import numpy as np
import pytest

from tests.helpers import conf_kwargs
from vortex_b200 import native as N
from vortex_b200 import profiles

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("P", [20, 32, 33, 129, 520])
@pytest.mark.parametrize("n", [1, 7, 8, 9, 127, 128, 129, 1000, 3001, 20000, 150000])
def test_birth_lanes(n, P):
    rng = np.random.default_rng(n + P)
    r, th = rng.uniform(0.6, 1.2, n), rng.uniform(0.0, 2 * math.pi, n)
    x, y, g = r * np.cos(th), r * np.sin(th), rng.normal(0.0, 1e-3, n)
    born = []
    for form in (N.PREC_FP64, N.PREC_FP32):
        sim = N.Sim(N.default_conf(**conf_kwargs(P, precision=form)), profiles.circle(P))
        sim.set_particles(x, y, g)
        sim.stage("birth")
        born.append(sim.particles()[2][n:])
        sim.close()
    assert len(born[0]) == len(born[1]) == P
    assert np.abs(born[1] - born[0]).max() <= 1e-5 * np.abs(born[0]).max()
