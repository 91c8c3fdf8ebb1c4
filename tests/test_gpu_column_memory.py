"""The standalone columns give their device memory back: a call with large
arrays leaves at most 64 MB with the process, and nothing with the pool of
the contexts. Measured in a child process, whose pools start empty."""
import subprocess
import sys
import os

import pytest

pytestmark = pytest.mark.gpu

CHILD = """
import sys
sys.path.insert(0, %r)
import numpy as np, torch, threading
import illum_gb300 as ig
from illum_gb300 import meshgen

def call(ncol, nz=40):
    g = np.random.default_rng(ncol)
    z = meshgen.geometric_depths(nz)
    T = np.asfortranarray(g.uniform(150.0, 250.0, (nz, ncol)))
    return ig.conductionQ_batch(z, 30.0, np.full(ncol, 50.0), np.full(ncol, 60.0), T, np.full(nz, 300.0),
                                np.full(nz, 1.05e6), 0.95, g.uniform(150.0, 250.0, ncol), bc_mode=ig.BC_NEWTON)

a = call(1000)
free0 = torch.cuda.mem_get_info()[0]
big = call(1 << 20)                      # 2 x 335 MB on the device
b = call(1000)
assert all(np.array_equal(x, y) for x, y in zip(a, b))
free1 = torch.cuda.mem_get_info()[0]
assert ig.device_pool_high()[0] == 0     # nothing from the contexts' pool
# several threads at once: the same results, and no more kept
out = [None] * 6
def work(k): out[k] = call(200000 + (k %% 2))
ts = [threading.Thread(target=work, args=(k,)) for k in range(6)]
[t.start() for t in ts]; [t.join() for t in ts]
for k in range(2, 6):
    assert all(np.array_equal(x, y) for x, y in zip(out[k], out[k %% 2]))
free2 = torch.cuda.mem_get_info()[0]
print("kept", (free0 - free1) >> 20, (free0 - free2) >> 20)
assert free0 - free1 <= (80 << 20) and free0 - free2 <= (80 << 20)
"""


def test_memory_goes_back(ilg):
    root = os.path.dirname(os.path.dirname(os.path.abspath(ilg.__file__)))
    r = subprocess.run([sys.executable, "-c", CHILD % root], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
