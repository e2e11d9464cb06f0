"""What the cell calls and the offline ECG keep between calls (a stream, a device and a
host block per thread): in a new thread, over the change from ordinary to pinned memory,
with sizes that grow and shrink, and after the program reset the device, when another
allocation may have the old block's address."""
import subprocess
import sys
import threading

import numpy as np
import pytest

from test_gpu_mahajan_groups import REST
from ucla_cmg_b200 import capi
from ucla_cmg_b200.simulation import ionic_step

pytestmark = pytest.mark.gpu

RESET = r"""
import ctypes, glob, os, sys
import numpy as np
sys.path.insert(0, {root!r})
import torch
from ucla_cmg_b200 import capi
from ucla_cmg_b200.simulation import ionic_step
rt = ctypes.CDLL(sorted(glob.glob(os.path.join(os.path.dirname(torch.__file__), "..", "nvidia", "cuda_runtime", "lib",
                                               "libcudart.so*")) + glob.glob("/usr/local/cuda/lib64/libcudart.so*"))[0])
def cells():
    S = np.tile(np.array({rest}), (500, 1))
    return ionic_step(capi.MAHAJAN, np.linspace(-85.0, -60.0, 500), 0.0, S, 0.01), S
first = [cells() for _ in range({calls})][0]
assert rt.cudaDeviceReset() == 0
# whatever lies at the old block's address belongs to somebody else now
size, blocks = 1 << 20, []
for _ in range(64):
    p = ctypes.c_void_p()
    assert rt.cudaMalloc(ctypes.byref(p), ctypes.c_size_t(size)) == 0
    assert rt.cudaMemset(p, 0x5a, ctypes.c_size_t(size)) == 0
    blocks.append(p)
again = cells()
assert all(np.array_equal(a, b) for a, b in zip(first, again))
for p in blocks:
    h = np.zeros(size, np.uint8)
    assert rt.cudaMemcpy(h.ctypes.data_as(ctypes.c_void_p), p, ctypes.c_size_t(size), 2) == 0
    assert (h == 0x5a).all()
print("as it was")
"""


@pytest.mark.parametrize("calls", [1, 9])          # ordinary and pinned host memory
def test_after_a_device_reset(gpu, calls):
    from conftest import ROOT
    r = subprocess.run([sys.executable, "-c", RESET.format(root=ROOT, calls=calls, rest=REST.tolist())], capture_output=True, text=True,
                       timeout=120)
    assert r.returncode == 0 and "as it was" in r.stdout, r.stdout + r.stderr


def test_threads_sizes_and_pinning(gpu):
    rng = np.random.default_rng(3)

    def call(n, V):
        S = np.tile(REST, (n, 1))
        return ionic_step(capi.MAHAJAN, V[:n], 0.0, S, 0.01), S

    V = rng.uniform(-85.0, -60.0, 200000)
    ref = call(200000, V)                           # two chunks
    bad = []

    def work():
        for n in (1, 300, 50, 7, 20000, 20, 9000, 140000, 3, 200000, 31):
            dv, S = call(n, V)
            if not (np.array_equal(dv, ref[0][:n]) and np.array_equal(S, ref[1][:n])):
                bad.append(n)

    threads = [threading.Thread(target=work) for _ in range(3)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad
