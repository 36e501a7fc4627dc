"""Bodies made after the caller reset the device (cudaDeviceReset, no body
left open, or one that was lost with it): the same bits as before it.  Covers
what the library keeps between bodies, the scalars' host copies and the
shared memory that kernels ask for: 1000 panels (over 48 KB in the panel
system's inverse), both pivot rules, expansions of order 20.  In a process of
its own, which ends with the lost body still open."""
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

CODE = """
import os, sys
import numpy as np
from tests.helpers import conf_kwargs, wake_cloud
from vortex_b200 import native as N
from vortex_b200 import profiles

def run(keep):
    out = []
    for pivot in (0, 1):
        kw = conf_kwargs(1000, precision=N.PREC_FP32, fmm_p=20, gj_pivot=pivot)
        sim = N.Sim(N.default_conf(**kw), profiles.circle(1000))
        sim.set_particles(*wake_cloud(3000, seed=1))
        sim.stage("velocity", "diffusion")
        sim.step(2)
        out += [np.array(a) for a in sim.particles()] + [sim.forces(), sim.matrix()]
        if keep:
            lost.append(sim)
        else:
            sim.close()
    return out

lost = []
first = run(False)
for keep in (False, True, False):
    assert N.cudart().cudaDeviceReset() == 0
    again = run(keep)
    assert all(np.array_equal(a, b) for a, b in zip(first, again))
assert len(lost) == 2
print("same")
sys.stdout.flush()
os._exit(0)
"""


def test_bodies_after_a_reset():
    r = subprocess.run([sys.executable, "-c", CODE], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout.strip() == "same", r.stdout[-500:] + r.stderr[-2000:]
