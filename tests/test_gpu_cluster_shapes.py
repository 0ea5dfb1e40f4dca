"""Swendsen-Wang and Wolff on every tile shape at its edges: lattices of one flat
tile and one site more, short rows on flat and narrow tiles, few rows on wide and
small ones, block tiles at 3D sizes one below, at and above theirs, extents of 1
and 2 along any direction, both streams; states, labels and sizes are the
oracle's.  Wolff on the few CTAs of a hot coupling, with the large first clusters
of a cold start."""
import numpy as np
import pytest

import plaquette_b200 as plq
from tests.test_gpu_cluster import _chain, _model, gpu  # noqa: F401  (gpu: the fixture)

pytestmark = pytest.mark.gpu

SHAPES = [
    (32, 32), (41, 25), (2, 16384), (3, 11000), (8, 4098), (4, 300), (1, 33000),         # flat, short rows
    (33, 20000), (12, 80000), (96, 7000), (64, 9500), (31, 30000),                       # narrow
    (140000, 8), (530000, 2), (70000, 16), (4096, 2), (1030, 5),                         # wide, few rows
    (64, 32, 32), (65, 33, 31), (63, 70, 40), (33, 17, 9), (31, 41, 17), (127, 62, 66),  # blocks
    (2, 2, 300), (4, 40, 30), (3, 70, 80), (8, 200, 180), (300, 2, 2), (257, 1, 3), (90, 80, 4), (5, 1, 1, 210000),
    (4, 5, 6, 20), (2, 3, 2, 3, 2, 3, 2), (1100, 1), (1, 1, 1, 1200),
]
IDS = [",".join(map(str, s)) for s in SHAPES]


def _beta(shape):
    return {1: 0.9, 2: 0.45}.get(sum(L > 2 for L in shape), 0.24)


@pytest.mark.parametrize("shape", SHAPES, ids=IDS)
def test_keyed(oracle, gpu, shape):  # noqa: F811
    lat, model, beta = oracle.Lattice(shape), _model(oracle, plq.ISING, 2), _beta(shape)
    start, _ = plq.hot_start(19, 2, lat.n_sites)
    chain = _chain(gpu, plq.ISING, 2, shape, plq.EXTENT_ALL, plq.RELABEL_REDRAW, beta, 19, start, plq.RNG_KEYED)
    want = start.copy()
    for sweep in range(3):
        roots = oracle.keyed_cluster_sweep(model, lat, want, oracle.ALL, plq.RELABEL_REDRAW, beta, oracle.fold_seed(19), sweep,
                                           want_roots=True)
        assert np.array_equal(next(chain), want), sweep
    assert np.array_equal(chain.labels(), roots)
    sizes = np.bincount(roots)
    hist = np.bincount(np.floor(np.log2(sizes[sizes > 0])).astype(int), minlength=32)[:32]
    assert np.array_equal(chain.size_histogram(), hist)
    chain.close()


@pytest.mark.parametrize("shape", SHAPES, ids=IDS)
def test_stream(oracle, gpu, shape):  # noqa: F811
    q, beta = 3, 1.6 * _beta(shape)
    lat, model = oracle.Lattice(shape), _model(oracle, plq.POTTS, q)
    start, off = plq.hot_start(20, q, lat.n_sites)
    chain = _chain(gpu, plq.POTTS, q, shape, plq.EXTENT_ALL, plq.RELABEL_FORCED, beta, 20, start, plq.RNG_STREAM, off)
    r = oracle.PcgStream(20)
    r.advance(off)
    want = start.copy()
    for sweep in range(2):
        probe = oracle.PcgStream(state=r.r.state, inc=r.r.inc)
        labels, _ = oracle.site_clusters(lat, want, model.bond_probability(beta), probe)
        oracle.cluster_sweep(model, lat, want, oracle.ALL, plq.RELABEL_FORCED, beta, r)
        assert np.array_equal(next(chain), want), sweep
        assert chain.stream_position() == r.draws
    # (ranked, the minimum sites are site_clusters' first-encounter numbers)
    assert np.array_equal(np.unique(chain.labels(), return_inverse=True)[1], labels)
    chain.close()


WOLFF = [(plq.ISING, 2, s, 1.1 * _beta(s)) for s in
         [(32, 32), (41, 25), (8, 4098), (33, 20000), (140000, 8), (65, 33, 31), (8, 200, 180), (300, 2, 2), (4, 5, 6, 20)]]
WOLFF += [(plq.POTTS, 20, (200, 300), 0.9), (plq.POTTS, 20, (40, 40, 40), 0.5), (plq.ISING, 2, (40, 50, 60), 0.1)]


@pytest.mark.parametrize("case", WOLFF, ids=lambda c: f"{c[0]}-{c[1]}-{'x'.join(map(str, c[2]))}")
def test_wolff(oracle, gpu, case):  # noqa: F811
    kind, q, shape, beta = case
    lat, model = oracle.Lattice(shape), _model(oracle, kind, q)
    start = np.zeros(lat.n_sites, np.uint8) if q > 2 else plq.hot_start(22, q, lat.n_sites)[0]
    chain = _chain(gpu, kind, q, shape, plq.EXTENT_SEEDED, plq.RELABEL_FORCED, beta, 22, start, plq.RNG_KEYED)
    chain.advance(8)
    want = start.copy()
    for t in range(8):
        oracle.keyed_cluster_sweep(model, lat, want, oracle.SEEDED, plq.RELABEL_FORCED, beta, oracle.fold_seed(22), t)
    assert np.array_equal(chain.read(), want)
    chain.close()
