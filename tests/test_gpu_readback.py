"""Large read-backs (plq_readback.cu): configurations above the staging threshold
whose size is no multiple of a piece come back whole, through read and next_batch,
from several threads at once and into a target of the caller's."""
import ctypes as C
import threading

import numpy as np
import pytest

import plaquette_b200 as plq

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(512, 250, 264), (130, 514, 504)], ids=lambda s: "x".join(map(str, s)))
def test_large_reads(shape):
    gpu = plq.Gpu.new()
    n = int(np.prod(shape))
    assert n > 32 << 20 and n % (1 << 20)
    start = np.random.default_rng(3).integers(0, 2, n, dtype=np.uint8)
    d = plq.make_desc(plq.ISING, 2, shape, plq.METROPOLIS, beta=0.2, seed=1, rng=plq.RNG_KEYED, sweeps_between=0, batch=1)
    chains = [plq.GpuChain(gpu, d, start) for _ in range(3)]
    got = [None] * 3

    def read(k):
        got[k] = chains[k].read()

    threads = [threading.Thread(target=read, args=(k,)) for k in range(3)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert all(np.array_equal(g, start) for g in got)
    states, _ = chains[0].next_batch(2)
    assert np.array_equal(states[0], start) and np.array_equal(states[1], start)
    out = np.full(n + 2, 9, np.uint8)
    plq.check(plq.lib().plq_chain_read(chains[0]._h, C.c_void_p(out.ctypes.data + 1)))
    assert out[0] == out[-1] == 9 and np.array_equal(out[1:-1], start)
