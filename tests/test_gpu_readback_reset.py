"""The pinned buffers of large read-backs end with the context: a program that
drops its chains and its context and resets the device (in a process of its own
here) can go on with a new one."""
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

PROGRAM = """
import ctypes, sys
sys.path.insert(0, sys.argv[1])
import numpy as np
import plaquette_b200 as plq

shape = (512, 300, 300)
start = np.random.default_rng(4).integers(0, 2, int(np.prod(shape)), dtype=np.uint8)
for k in range(3):
    gpu = plq.Gpu.new()
    d = plq.make_desc(plq.ISING, 2, shape, plq.METROPOLIS, beta=0.2, seed=1, rng=plq.RNG_KEYED, batch=1)
    chain = plq.GpuChain(gpu, d, start)
    assert np.array_equal(chain.read(), start)
    chain.close()
    del chain, gpu
    assert ctypes.CDLL("libcudart.so.12").cudaDeviceReset() == 0
print("done")
"""


def test_reset_between_contexts():
    import plaquette_b200

    root = plaquette_b200.__path__[0].rsplit("/", 1)[0]
    r = subprocess.run([sys.executable, "-c", PROGRAM, root], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip() == "done", r.stderr[-2000:]
