"""Swendsen-Wang labels and states at the edges of the labelling tiles: extents
one below, at and one above a tile's, tiles that overhang in every direction,
small and large tiles (the large ones from two CTAs per SM on), directions past
the tile's, all bonds closed and all open, both streams; labels and sizes are
those of the oracle, asked for before, between and after sweeps."""
import numpy as np
import pytest

import plaquette_b200 as plq
from tests.test_gpu_cluster import _chain, _compact, _model, gpu  # noqa: F401  (gpu: the fixture)

pytestmark = pytest.mark.gpu

SHAPES = [
    (1,), (31,), (257,), (1000,),
    (127, 15), (128, 16), (129, 17), (33, 65), (1, 40), (2, 2),
    (31, 7, 3), (32, 8, 4), (33, 9, 5), (70, 6, 11), (1, 3, 9),
    (34, 9, 5, 3), (3, 2, 3, 2, 3),
    (1031, 1203), (131, 97, 101), (40, 18, 33, 50),  # large tiles
]
CASES = [(plq.ISING, 2, 0.45, plq.RELABEL_REDRAW), (plq.POTTS, 3, 0.9, plq.RELABEL_FORCED)]


@pytest.mark.parametrize("kind,q,beta,relabel", CASES, ids=["ising", "potts3-forced"])
@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s)))
def test_keyed(oracle, gpu, shape, kind, q, beta, relabel):  # noqa: F811
    lat = oracle.Lattice(shape)
    model = _model(oracle, kind, q)
    start, _ = plq.hot_start(9, q, lat.n_sites)
    beta = beta if len(shape) < 3 else beta / 2
    chain = _chain(gpu, kind, q, shape, plq.EXTENT_ALL, relabel, beta, 9, start, plq.RNG_KEYED)
    want = start.copy()
    for sweep in range(3):
        roots = oracle.keyed_cluster_sweep(model, lat, want, oracle.ALL, relabel, beta, oracle.fold_seed(9), sweep,
                                           want_roots=True)
        assert np.array_equal(next(chain), want), sweep
        if sweep != 1:
            sizes = np.bincount(roots)
            hist = np.bincount(np.floor(np.log2(sizes[sizes > 0])).astype(int), minlength=32)[:32]
            if sweep == 0:
                assert np.array_equal(chain.size_histogram(), hist)
            assert np.array_equal(chain.labels(), roots), sweep
            assert np.array_equal(chain.size_histogram(), hist)


@pytest.mark.parametrize("shape", [(129, 17), (33, 9, 5), (34, 9, 5, 3), (1031, 1203), (131, 97, 101)],
                         ids=lambda s: "x".join(map(str, s)))
def test_stream(oracle, gpu, shape):  # noqa: F811
    kind, q, relabel = plq.POTTS, 5, plq.RELABEL_FORCED
    beta = 1.17 if len(shape) == 2 else 0.6
    lat = oracle.Lattice(shape)
    model = _model(oracle, kind, q)
    start, off = plq.hot_start(10, q, lat.n_sites)
    chain = _chain(gpu, kind, q, shape, plq.EXTENT_ALL, relabel, beta, 10, start, plq.RNG_STREAM, off)
    r = oracle.PcgStream(10)
    r.advance(off)
    want = start.copy()
    for sweep in range(2):
        probe = oracle.PcgStream(state=r.r.state, inc=r.r.inc)
        labels, _ = oracle.site_clusters(lat, want, model.bond_probability(beta), probe)
        oracle.cluster_sweep(model, lat, want, oracle.ALL, relabel, beta, r)
        assert np.array_equal(next(chain), want), sweep
        assert chain.stream_position() == r.draws
        assert np.array_equal(_compact(chain.labels()), labels)


@pytest.mark.parametrize("beta", [0.0, 50.0], ids=["closed", "open"])
@pytest.mark.parametrize("shape", [(129, 17), (33, 9, 5), (1031, 1203)], ids=lambda s: "x".join(map(str, s)))
def test_all_or_no_bonds(gpu, shape, beta):  # noqa: F811
    n = int(np.prod(shape))
    chain = _chain(gpu, plq.ISING, 2, shape, plq.EXTENT_ALL, plq.RELABEL_REDRAW, beta, 3, np.zeros(n, np.uint8),
                   plq.RNG_KEYED)
    next(chain)
    assert np.array_equal(chain.labels(), np.arange(n) if beta == 0.0 else np.zeros(n))


WOLFF = [
    (plq.ISING, 2, (31,), 1.0, plq.RELABEL_FORCED), (plq.ISING, 2, (2, 2), 0.4, plq.RELABEL_FORCED),
    (plq.ISING, 2, (129, 17), 0.2, plq.RELABEL_FORCED),      # small clusters: growth alone
    (plq.ISING, 2, (129, 17), 0.44, plq.RELABEL_REDRAW),     # ... ended after the call
    (plq.POTTS, 3, (64, 96), 1.005, plq.RELABEL_FORCED),     # ... and the decomposition
    (plq.ISING, 2, (33, 9, 5), 0.25, plq.RELABEL_FORCED), (plq.POTTS, 4, (34, 9, 5, 3), 0.5, plq.RELABEL_REDRAW),
    (plq.ISING, 2, (33, 9, 5), 50.0, plq.RELABEL_FORCED), (plq.ISING, 2, (33, 9, 5), 0.0, plq.RELABEL_FORCED),
    (plq.ISING, 2, (401, 307), 0.47, plq.RELABEL_FORCED),
]


@pytest.mark.parametrize("case", WOLFF, ids=lambda c: f"{c[0]}-{c[1]}-{'x'.join(map(str, c[2]))}-{c[3]}-{c[4]}")
def test_wolff(oracle, gpu, case):  # noqa: F811
    """Growth alone, growth that ends after the call and the decomposition give the seeded filter's
    states and cluster size, one update a launch and many in one."""
    kind, q, shape, beta, relabel = case
    lat = oracle.Lattice(shape)
    model = _model(oracle, kind, q)
    start, _ = plq.hot_start(12, q, lat.n_sites)
    args = (gpu, kind, q, shape, plq.EXTENT_SEEDED, relabel, beta, 12, start, plq.RNG_KEYED)
    one, many = _chain(*args), _chain(*args)
    updates = 12
    many.advance(updates)
    want = start.copy()
    for t in range(updates):
        before = want.copy()
        oracle.keyed_cluster_sweep(model, lat, want, oracle.SEEDED, relabel, beta, oracle.fold_seed(12), t)
        assert np.array_equal(next(one), want), t
        if relabel == plq.RELABEL_FORCED:
            flipped = int((before != want).sum())
            assert one.size_histogram()[flipped.bit_length() - 1] == 1
    assert np.array_equal(many.read(), want)
