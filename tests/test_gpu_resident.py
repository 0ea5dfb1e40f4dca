"""Resident launches (plq_resident.cu) against the per-pass kernels, which the
other tests hold to the oracle: final configurations, every sample's bytes and
primaries and the stream position are the same, at the edges of the shares (one
CTA, a cluster, a grid, several words a thread), of the words (rows of 2 to 130
sites, links to 64 a row) and for every other chain that runs resident; calls may
be mixed, and chains of several host threads run side by side."""
import threading

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


def _pair(gpu, kind, q, shape, kernel, rng, beta, **kw):
    n = int(np.prod(shape)) * (len(shape) if kind == plq.GAUGE else 1)
    start, off = plq.hot_start(21, q, n)
    args = dict(beta=beta, seed=21, rng=rng, stream_offset=off if rng == plq.RNG_STREAM else 0, batch=1, **kw)
    return [plq.GpuChain(gpu, plq.make_desc(kind, q, shape, kernel, flags=flags, **args), start)
            for flags in (0, plq.FLAG_GENERIC_PASS)]


def _check(a, b):
    a.advance(2)
    b.advance(2)
    sa, pa = a.next_batch(3)
    sb, pb = b.next_batch(3)
    assert np.array_equal(sa, sb) and np.array_equal(pa, pb)
    _, pa = a.next_batch(2, states=False)
    _, pb = b.next_batch(2, states=False)
    assert np.array_equal(pa, pb)
    a.advance(1)
    b.advance(1)
    assert np.array_equal(a.read(), b.read())
    assert a.sweeps_done == b.sweeps_done
    if a.desc.rng == plq.RNG_STREAM:
        assert a.stream_position() == b.stream_position()


SITES = [(2, 2), (4, 6), (30, 8), (32, 10), (62, 6), (64, 64), (66, 12), (128, 10), (130, 34), (190, 46), (64, 130),
         (2, 4, 6), (16, 14, 12), (34, 16, 10), (48, 40, 36), (64, 24, 22), (66, 30, 28), (126, 50, 20), (200, 60, 60),
         (1026, 514), (64, 128, 132)]


@pytest.mark.parametrize("kernel", [plq.METROPOLIS, plq.HEATBATH], ids=["metro", "hb"])
@pytest.mark.parametrize("shape", SITES, ids=lambda s: "x".join(map(str, s)))
def test_packed_sites(gpu, shape, kernel):
    beta = 0.44 if len(shape) == 2 else 0.22
    _check(*_pair(gpu, plq.ISING, 2, shape, kernel, plq.RNG_KEYED, beta, h=0.1, sweeps_between=2))


@pytest.mark.parametrize("shape", [(6, 4), (66, 12), (34, 16, 10)], ids=lambda s: "x".join(map(str, s)))
def test_packed_potts2(gpu, shape):
    _check(*_pair(gpu, plq.POTTS, 2, shape, plq.HEATBATH, plq.RNG_KEYED, 0.6, sweeps_between=1))


LINKS = [(2, 2), (18, 6), (64, 4), (2, 4, 2), (16, 6, 4), (34, 10, 8), (62, 4, 4), (64, 40, 38), (4, 4, 4, 4), (6, 4, 2, 4),
         (16, 8, 6, 4), (24, 16, 14, 12), (40, 6, 4, 6), (32, 24, 24, 24)]


@pytest.mark.parametrize("kernel", [plq.METROPOLIS, plq.HEATBATH], ids=["metro", "hb"])
@pytest.mark.parametrize("shape", LINKS, ids=lambda s: "x".join(map(str, s)))
def test_packed_links(gpu, shape, kernel):
    _check(*_pair(gpu, plq.GAUGE, 2, shape, kernel, plq.RNG_KEYED, {2: 0.7, 3: 0.76, 4: 0.44}[len(shape)],
                  sweeps_between=2))


OTHERS = [  # kind, q, shape, kernel, rng
    (plq.POTTS, 5, (102, 50), plq.METROPOLIS, plq.RNG_KEYED), (plq.POTTS, 3, (8, 6, 4), plq.METROPOLIS, plq.RNG_KEYED),
    (plq.POTTS, 4, (4, 2, 4, 6), plq.METROPOLIS, plq.RNG_KEYED), (plq.POTTS, 3, (10,), plq.METROPOLIS, plq.RNG_KEYED),
    (plq.POTTS, 3, (30, 26, 22), plq.HEATBATH, plq.RNG_KEYED), (plq.POTTS, 7, (34, 30), plq.HEATBATH, plq.RNG_KEYED),
    (plq.POTTS, 3, (64, 60, 36), plq.HEATBATH, plq.RNG_KEYED), (plq.POTTS, 4, (32, 20, 12), plq.HEATBATH, plq.RNG_STREAM),
    (plq.POTTS, 5, (62, 56), plq.HEATBATH, plq.RNG_STREAM), (plq.ISING, 2, (40, 36, 30), plq.HEATBATH, plq.RNG_STREAM),
    (plq.ISING, 2, (32,), plq.METROPOLIS, plq.RNG_KEYED), (plq.ISING, 2, (6, 4, 4, 2), plq.METROPOLIS, plq.RNG_KEYED),
    (plq.ISING, 2, (8, 4, 4, 6), plq.HEATBATH, plq.RNG_KEYED), (plq.GAUGE, 2, (16, 12, 10), plq.HEATBATH, plq.RNG_STREAM),
    (plq.GAUGE, 2, (6, 4, 6, 4), plq.HEATBATH, plq.RNG_STREAM), (plq.GAUGE, 2, (70, 6, 4), plq.METROPOLIS, plq.RNG_KEYED),
    (plq.POTTS, 6, (1002, 750), plq.METROPOLIS, plq.RNG_KEYED),
]


@pytest.mark.parametrize("case", OTHERS, ids=lambda c: f"{c[0]}-{c[1]}-{'x'.join(map(str, c[2]))}-{c[3]}-{c[4]}")
def test_bytes(gpu, case):
    kind, q, shape, kernel, rng = case
    _check(*_pair(gpu, kind, q, shape, kernel, rng, 0.6, sweeps_between=2))


def test_no_sweeps_between_samples(gpu):
    a, _ = _pair(gpu, plq.ISING, 2, (20, 6), plq.METROPOLIS, plq.RNG_KEYED, 0.4, sweeps_between=0)
    start = a.read()
    states, prim = a.next_batch(2)
    assert np.array_equal(states, np.stack([start, start])) and np.array_equal(prim[0], a.primaries())


def test_chains_of_several_threads(gpu):
    """Grids of chains on their own streams, launched from four threads at once."""
    shapes = [(200, 60, 60), (66, 30, 28), (24, 16, 14, 12), (512, 512)]
    pairs = [_pair(gpu, plq.GAUGE if len(s) == 4 else plq.ISING, 2, s, plq.HEATBATH, plq.RNG_KEYED, 0.3) for s in shapes]

    def run(chain):
        for _ in range(20):
            chain.advance(5)
        chain.sync()

    threads = [threading.Thread(target=run, args=(p[0],)) for p in pairs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for a, b in pairs:
        b.advance(100)
        assert np.array_equal(a.read(), b.read())


@pytest.mark.parametrize("kernel", [plq.METROPOLIS, plq.HEATBATH], ids=["metro", "hb"])
@pytest.mark.parametrize("shape", SITES + [(256, 250), (512, 190, 40)], ids=lambda s: "x".join(map(str, s)))
def test_stream_sites(gpu, shape, kernel):
    beta = 0.44 if len(shape) == 2 else 0.22
    _check(*_pair(gpu, plq.ISING, 2, shape, kernel, plq.RNG_STREAM, beta, h=0.1, sweeps_between=2))


@pytest.mark.parametrize("kernel", [plq.METROPOLIS, plq.HEATBATH], ids=["metro", "hb"])
@pytest.mark.parametrize("shape", LINKS, ids=lambda s: "x".join(map(str, s)))
def test_stream_links(gpu, shape, kernel):
    _check(*_pair(gpu, plq.GAUGE, 2, shape, kernel, plq.RNG_STREAM, {2: 0.7, 3: 0.76, 4: 0.44}[len(shape)],
                  sweeps_between=2))


@pytest.mark.parametrize("beta", [0.0, 0.7, 300.0])
@pytest.mark.parametrize("shape", [(8, 6), (66, 12), (130, 60, 22)], ids=lambda s: "x".join(map(str, s)))
def test_stream_extreme_couplings(gpu, shape, beta):
    """No variable draws (beta = 0: every move is downhill), probabilities of 0 (cut points of 0)."""
    _check(*_pair(gpu, plq.POTTS, 2, shape, plq.METROPOLIS, plq.RNG_STREAM, beta, sweeps_between=1))
