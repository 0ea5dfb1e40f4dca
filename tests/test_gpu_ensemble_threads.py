"""An ensemble's members read from several host threads at once: link members go
to the host through one staging buffer, and each call gets its own member's bytes."""
import threading

import numpy as np
import pytest

import plaquette_b200 as plq
from plaquette_b200.ensemble import Ensemble

pytestmark = pytest.mark.gpu


def test_members_read_from_several_threads():
    gpu = plq.Gpu.new()
    if gpu is None:
        pytest.fail("no CUDA device")
    shapes = [(8, 8, 8, 8), (6, 4, 4, 4), (10, 8, 8, 8), (4, 4, 4, 4)]
    descs, starts = [], []
    for i, shape in enumerate(shapes):
        start, _ = plq.hot_start(70 + i, 2, 4 * int(np.prod(shape)))
        descs.append(plq.make_desc(plq.GAUGE, 2, shape, plq.HEATBATH, beta=0.44, seed=70 + i, rng=plq.RNG_KEYED, batch=1))
        starts.append(start)
    ens = Ensemble(gpu, descs, starts)
    bad = []

    def read(m):
        for _ in range(200):
            if not np.array_equal(ens.read(m), starts[m]):
                bad.append(m)

    threads = [threading.Thread(target=read, args=(m,)) for m in range(len(shapes))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad
