"""Served jobs' packed rows live in what the budget leaves beside the bytes on
which jobs are admitted: a job that fits the budget is admitted at once, though
the rows of a running one fill it, and both results are those of the jobs alone."""
import time

import numpy as np
import pytest

import plaquette_b200 as plq
from plaquette_b200.serving import JOB_ACTIVE, JOB_DONE, Server

pytestmark = pytest.mark.gpu


def test_rows_make_room_for_a_queued_job():
    gpu = plq.Gpu.new()
    if gpu is None:
        pytest.fail("no CUDA device")
    shape = (4, 256, 256)  # rows of four sites: 32-bit rows are as large as the bytes
    n = int(np.prod(shape))

    def job(seed):
        start, _ = plq.hot_start(seed, 2, n)
        return plq.make_desc(plq.ISING, 2, shape, plq.METROPOLIS, beta=0.3, seed=seed, rng=plq.RNG_KEYED, batch=1), start

    srv = Server(gpu, 2 * n + 16384, 8, 2.0)
    sweeps = 60000
    a = srv.submit(*job(5), sweeps, want_states=True)
    for _ in range(2000):
        if srv.stats()["running"]:
            break
        time.sleep(0.001)
    time.sleep(0.02)
    assert srv.stats()["device_bytes"] > 2 * n  # its rows have the rest of the budget
    b = srv.submit(*job(6), 5, want_states=True)
    assert srv.wait(b, 60.0) == JOB_DONE
    assert srv.wait(a, 0.0) == JOB_ACTIVE
    assert srv.wait(a, 60.0) == JOB_DONE
    for jid, seed, k in ((a, 5, sweeps), (b, 6, 5)):
        alone = plq.GpuChain(gpu, *job(seed))
        alone.advance(k)
        states, prim, _ = srv.result(jid, states=True)
        assert np.array_equal(states, alone.read())
        assert list(prim) == list(alone.primaries())
    srv.close()
