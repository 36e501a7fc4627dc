"""Device memory after bodies are closed: with the last one (one that could
not be made, or a batch's members, too) the device's pool holds what it held
before the first, so that a plain cudaMalloc can have all of it.  In a process of its
own: another test's open body would keep its memory."""
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

CODE = """
import ctypes as C
from tests.helpers import conf_kwargs, wake_cloud
from vortex_b200 import native as N
from vortex_b200 import profiles

rt = N.cudart()
pool = C.c_void_p()

def held():
    assert rt.cudaDeviceGetDefaultMemPool(C.byref(pool), 0) == 0
    v = C.c_uint64()
    assert rt.cudaMemPoolGetAttribute(pool, 5, C.byref(v)) == 0   # bytes the pool has of the device's
    return v.value

def body(n, **kw):
    sim = N.Sim(N.default_conf(**conf_kwargs(200, precision=N.PREC_FP32, **kw)), profiles.circle(200))
    sim.set_particles(*wake_cloud(n, seed=1))
    sim.step(1)
    return sim

assert held() == 0
body(1000).close()
assert held() == 0
a, b, c = body(300000), body(1000), body(20000)
b.close()
a.close()
c.count()
assert held() > 0
c.close()
assert held() == 0
members = [body(1000), body(2000)]
batch = N.Batch(members)
batch.step(2)
batch.sync()
batch.close()
for s in members:
    s.close()
assert held() == 0
pan = profiles.circle(200)
pan["right"] = pan["left"]       # no panel system
try:
    N.Sim(N.default_conf(**conf_kwargs(200)), pan)
    raise SystemExit("made")
except N.VxError:
    pass
assert held() == 0
print("given back")
"""


def test_pool_given_back():
    r = subprocess.run([sys.executable, "-c", CODE], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout.strip() == "given back", r.stdout[-500:] + r.stderr[-2000:]
