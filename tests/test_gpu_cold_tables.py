"""Packed decisions at couplings so cold that a probability underflows to 0 (a
cut point of 0, which the open-draw comparison cannot express and the marked
table takes): chains equal the oracle's keyed sweeps, ensemble members their
own byte-pass chains.  The middle coupling has all of its cut points above 0."""
import numpy as np
import pytest

import plaquette_b200 as plq
from plaquette_b200.ensemble import Ensemble
from tests.test_gpu_local import run_pair

pytestmark = pytest.mark.gpu

BETAS = [0.0, 1.2, 60.0]
KERNELS = [plq.METROPOLIS, plq.HEATBATH]


@pytest.fixture(scope="module")
def gpu():
    g = plq.Gpu.new()
    if g is None:
        pytest.fail("no CUDA device")
    return g


@pytest.mark.parametrize("flags", [0, plq.FLAG_NO_FIRST_HASH], ids=["first-hash-array", "hashed"])
@pytest.mark.parametrize("beta", BETAS)
@pytest.mark.parametrize("kernel", KERNELS, ids=["metro", "hb"])
@pytest.mark.parametrize("shape", [(64, 6), (128, 4, 6)], ids=["2d", "3d"])
def test_chain(oracle, gpu, shape, kernel, beta, flags):
    got, want, chain, *_ = run_pair(oracle, gpu, plq.ISING, 2, shape, kernel, plq.RNG_KEYED, beta, 4, flags=flags)
    assert chain.path == "packed"
    assert np.array_equal(got, want)


@pytest.mark.parametrize("beta", BETAS)
@pytest.mark.parametrize("kernel", KERNELS, ids=["metro", "hb"])
def test_members(gpu, kernel, beta):
    shapes = [(plq.ISING, (20, 6, 4)), (plq.ISING, (64, 8)), (plq.GAUGE, (4, 4, 4, 4)), (plq.GAUGE, (6, 4, 4)),
              (plq.GAUGE, (18, 6))]
    descs, starts, chains = [], [], []
    for i, (kind, shape) in enumerate(shapes):
        n = int(np.prod(shape)) * (len(shape) if kind == plq.GAUGE else 1)
        start, _ = plq.hot_start(50 + i, 2, n)
        args = dict(beta=beta, seed=50 + i, rng=plq.RNG_KEYED, batch=1)
        descs.append(plq.make_desc(kind, 2, shape, kernel, **args))
        starts.append(start)
        chains.append(plq.GpuChain(gpu, plq.make_desc(kind, 2, shape, kernel, flags=plq.FLAG_GENERIC_PASS, **args),
                                   start))
    ens = Ensemble(gpu, descs, starts)
    ens.advance(4)
    for m, c in enumerate(chains):
        c.advance(4)
        assert np.array_equal(ens.read(m), c.read()), m
