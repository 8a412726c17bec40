"""Who sets the release threshold of the device's default memory pool: the first
call raises one that is 0, a threshold of the application's stands, and an
engine's budget is not undone by calls that start beside it.  Each case in a
process of its own, since the first call on a device decides."""
import subprocess
import sys
from pathlib import Path

import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

ROOT = Path(__file__).resolve().parent.parent

PRELUDE = """
import ctypes as C, sys, threading
sys.path[:0] = [%r, %r]
import conftest, torch
from oxideav_av1_b200 import abi, engine, postfilter, synth
torch.cuda.init()
cu = C.CDLL("libcuda.so.1")
dev, pool = C.c_int(), C.c_void_p()
assert cu.cuDeviceGet(C.byref(dev), 0) == 0 and cu.cuDeviceGetDefaultMemPool(C.byref(pool), dev) == 0
RELEASE_THRESHOLD = 4  # CU_MEMPOOL_ATTR_RELEASE_THRESHOLD
def threshold(v=None):
    c = C.c_uint64(0 if v is None else v)
    f = cu.cuMemPoolGetAttribute if v is None else cu.cuMemPoolSetAttribute
    assert f(pool, RELEASE_THRESHOLD, C.byref(c)) == 0
    return c.value
d = postfilter.DeviceFrame(synth.make_frame(seed=701, width=64, height=64))
def call():
    torch.cuda.set_device(0)
    s = torch.cuda.Stream()
    postfilter.run_postfilter([d], stream=s)
    s.synchronize()
""" % (str(ROOT / "tests"), str(ROOT))


@pytest.mark.parametrize("body", [
    # the default of 0 is raised, once: what is set afterwards stands
    "assert threshold() == 0; call(); assert threshold() == 256 << 20; threshold(0); call(); assert threshold() == 0",
    # the application's own, 1 byte for none
    "threshold(1); call(); assert threshold() == 1",
    # an engine's budget, whatever calls run while it is made
    """
ts = [threading.Thread(target=call) for _ in range(6)]
for t in ts: t.start()
e = engine.Engine(device=0, budget_bytes=3 << 30)
for t in ts: t.join()
assert threshold() == 3 << 30
e.close()
""",
], ids=["raised once", "set by the application", "engine beside first calls"])
def test_release_threshold(body):
    r = subprocess.run([sys.executable, "-c", PRELUDE + body], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
