"""Calls longer than one launch takes (2^33 updates of a resident chain, 1024
updates of a Wolff chain): the pieces continue one another -- sweep counter, PCG
position, samples and their places -- and equal the per-pass kernels."""
import numpy as np
import pytest

import plaquette_b200 as plq

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gpu():
    g = plq.Gpu.new()
    if g is None:
        pytest.fail("no CUDA device")
    return g


@pytest.mark.parametrize("rng", [plq.RNG_KEYED, plq.RNG_STREAM], ids=["keyed", "stream"])
def test_resident(gpu, rng):
    shape = (250, 250, 250)  # 549 sweeps a launch
    start, off = plq.hot_start(31, 2, int(np.prod(shape)))
    out = []
    for flags in (0, plq.FLAG_NO_FIRST_HASH):
        d = plq.make_desc(plq.ISING, 2, shape, plq.METROPOLIS, beta=0.2216544, seed=31, rng=rng, stream_offset=off,
                          sweeps_between=300, batch=5, flags=flags)
        c = plq.GpuChain(gpu, d, start)
        assert c.resident == (flags == 0)
        before = c.launches
        c.advance(1200)
        c.sync()
        assert (c.launches - before == 3) == (flags == 0)
        batch = c.next_batch(3)  # one sample a launch
        out.append([batch[0], batch[1], c.sweeps_done, c.stream_position() if rng == plq.RNG_STREAM else 0])
        c.close()
    assert out[0][2] == 2100
    for a, b in zip(*out):
        assert np.array_equal(a, b)


def test_samples_further_apart_than_a_launch(gpu):
    shape = (250, 250, 250)
    start, _ = plq.hot_start(32, 2, int(np.prod(shape)))
    out = []
    for flags in (0, plq.FLAG_NO_FIRST_HASH):
        d = plq.make_desc(plq.ISING, 2, shape, plq.HEATBATH, beta=0.2216544, seed=32, rng=plq.RNG_KEYED, sweeps_between=700,
                          batch=2, flags=flags)
        c = plq.GpuChain(gpu, d, start)
        out.append(c.next_batch(2))
        c.close()
    assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])


def test_wolff(gpu):
    shape = (20, 18, 16)
    start, _ = plq.hot_start(33, 2, int(np.prod(shape)))
    d = plq.make_desc(plq.ISING, 2, shape, plq.CLUSTER, beta=0.23, seed=33, rng=plq.RNG_KEYED, sweeps_between=1, batch=1,
                      extent=plq.EXTENT_SEEDED, relabel=plq.RELABEL_FORCED)
    one, many = plq.GpuClusterChain(gpu, d, start), plq.GpuClusterChain(gpu, d, start)
    one.advance(2500)
    for _ in range(5):
        many.advance(500)
    assert np.array_equal(one.read(), many.read()) and one.sweeps_done == many.sweeps_done == 2500
