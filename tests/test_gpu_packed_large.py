"""The bit-packed passes that stream each site's first hash from memory, at the
sizes that take them (launches per pass; smaller lattices run resident): 2D and 3D,
rows of one, three and 64 words, word counts that are no multiple of the array's
32-word blocks, both updaters, and couplings so cold that the table is a marked
one -- against the byte passes of the same chain."""
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


@pytest.mark.parametrize("beta", [0.3, 60.0])
@pytest.mark.parametrize("kernel", [plq.METROPOLIS, plq.HEATBATH], ids=["metro", "hb"])
@pytest.mark.parametrize("shape", [(64, 512, 514), (192, 298, 294), (4096, 4098), (192, 87384)],
                         ids=lambda s: "x".join(map(str, s)))
def test_first_hash_passes(gpu, shape, kernel, beta):
    start, _ = plq.hot_start(61, 2, int(np.prod(shape)))
    out = []
    for flags in (0, plq.FLAG_NO_PACKED):
        d = plq.make_desc(plq.ISING, 2, shape, kernel, beta=beta, seed=61, rng=plq.RNG_KEYED, sweeps_between=3, batch=1,
                          flags=flags)
        c = plq.GpuChain(gpu, d, start)
        assert not c.resident and (c.path == "packed") == (flags == 0)
        c.advance(1)
        out.append(c.next_sample())
        c.close()
    assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])


@pytest.mark.parametrize("shape", [(64, 48), (66, 34), (130, 34), (48, 40, 36), (34, 30, 22), (512, 64, 32)],
                         ids=lambda s: "x".join(map(str, s)))
def test_lookback_passes(gpu, shape):
    """Metropolis on the PCG stream by the look-back passes, which a chain without packed words
    takes, equals the resident launch."""
    start, off = plq.hot_start(62, 2, int(np.prod(shape)))
    out = []
    for flags in (0, plq.FLAG_NO_PACKED):
        d = plq.make_desc(plq.ISING, 2, shape, plq.METROPOLIS, beta=0.4 if len(shape) == 2 else 0.22, seed=62,
                          rng=plq.RNG_STREAM, stream_offset=off, sweeps_between=5, batch=1, flags=flags)
        c = plq.GpuChain(gpu, d, start)
        assert c.path == "lookback" and c.resident == (flags == 0)
        out.append((c.next_sample(), c.stream_position()))
        c.close()
    assert np.array_equal(out[0][0][0], out[1][0][0]) and np.array_equal(out[0][0][1], out[1][0][1])
    assert out[0][1] == out[1][1]
