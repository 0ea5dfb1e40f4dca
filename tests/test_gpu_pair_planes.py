"""Axis pair sums at the sizes that count them on bit planes (smaller lattices
and long thin ones count bytes), against numpy: rows of whole words, of ragged
ones and shorter than a word, one to three planes, 1D to 4D; and, on the other
side of the line, lattices that count bytes."""
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


def _differing(shape, cfg):
    """Differing pairs per axis and displacement 1 .. L/2."""
    a = cfg.reshape(shape[::-1])
    return [[int((a != np.roll(a, -r, axis=len(shape) - 1 - mu)).sum()) for r in range(1, L // 2 + 1)]
            for mu, L in enumerate(shape)]


SHAPES = [(1024, 1024), (1002, 750), (100, 100, 100), (66, 130, 96), (30, 192, 190), (130, 66, 64), (256, 96, 62),
          (24, 24, 24, 24), (20000,),
          (64, 64), (2, 2048), (8, 8, 8, 8), (4, 256, 256), (1000,)]


@pytest.mark.parametrize("q", [2, 3, 5])
@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s)))
def test_pair_sums(gpu, shape, q):
    n = int(np.prod(shape))
    start = np.random.default_rng(8).integers(0, q, n, dtype=np.uint8)
    start[: n // 3] = 0  # (not alike in every direction)
    c = plq.GpuChain(gpu, plq.make_desc(plq.POTTS, q, shape, plq.HEATBATH, beta=0.5, seed=8, rng=plq.RNG_KEYED, batch=1),
                     start)
    got = c.axis_pair_sums()
    for mu, differ in enumerate(_differing(shape, start)):
        assert list(got[mu]) == [n] + [n - k for k in differ], mu
