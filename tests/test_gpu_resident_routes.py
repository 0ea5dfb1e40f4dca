"""Both sides of the lines between the resident launch of packed words and the
per-pass kernels on bytes (rows that fill little of a word, rows whose last word
is short, whole words), for both streams and updaters: the chain takes the side
the sizes name, and its states, primaries and stream position are those of the
generic passes."""
import numpy as np
import pytest

import plaquette_b200 as plq
from tests.test_gpu_resident import _check, _pair, gpu  # noqa: F401  (gpu: the fixture)

pytestmark = pytest.mark.gpu

M, H, K, S = plq.METROPOLIS, plq.HEATBATH, plq.RNG_KEYED, plq.RNG_STREAM
ROUTES = [  # kind, shape, updater, stream, resident
    (plq.ISING, (4, 1 << 19), M, K, False), (plq.ISING, (4, (1 << 19) - 2), M, K, True),
    (plq.ISING, (8, 1024, 512), H, K, False), (plq.ISING, (2, 1 << 20), H, K, False), (plq.ISING, (6, 1 << 19), M, K, True),
    (plq.ISING, (72, 116510), M, K, False), (plq.ISING, (72, 116508), H, K, True), (plq.ISING, (84, 116510), M, K, True),
    (plq.ISING, (4, 1 << 17), H, S, False), (plq.ISING, (4, (1 << 17) - 2), H, S, True),
    (plq.ISING, (8, 512, 512), H, S, False), (plq.ISING, (2, 1 << 19), H, S, False), (plq.ISING, (6, 1 << 19), H, S, True),
    (plq.ISING, (2, 163840), M, S, False), (plq.ISING, (2, 163838), M, S, True), (plq.ISING, (6, 512, 512), M, S, False),
    (plq.ISING, (16, 1 << 17), M, S, False), (plq.ISING, (16, (1 << 17) - 2), M, S, True),
    (plq.ISING, (32, 1 << 17), M, S, False), (plq.ISING, (80, 13108), M, S, False), (plq.ISING, (112, 9364), M, S, True),
    (plq.ISING, (64, 1 << 15), M, S, True), (plq.ISING, (8, 1 << 18), M, S, True),
    (plq.GAUGE, (2, 1 << 18), M, S, False), (plq.GAUGE, (2, (1 << 18) - 2), M, S, True), (plq.GAUGE, (4, 1024, 512), M, S, False),
    (plq.GAUGE, (4, 1 << 18), H, S, False), (plq.GAUGE, (8, 1 << 19), H, S, False), (plq.GAUGE, (8, 512, 1024), H, S, True),
    (plq.GAUGE, (4, 1 << 20), H, K, False), (plq.GAUGE, (2, 1 << 20), M, K, True),
    (plq.ISING, (4096, 4096), M, K, False), (plq.ISING, (4096, 4094), H, K, True),
]


@pytest.mark.parametrize("case", ROUTES, ids=lambda c: f"{c[0]}-{'x'.join(map(str, c[1]))}-{c[2]}-{c[3]}")
def test_route(gpu, case):  # noqa: F811
    kind, shape, updater, rng, resident = case
    a, b = _pair(gpu, kind, 2, shape, updater, rng, 0.4 if len(shape) == 2 else 0.22, sweeps_between=1)
    assert a.resident == resident and not b.resident
    _check(a, b)
    a.close()
    b.close()
