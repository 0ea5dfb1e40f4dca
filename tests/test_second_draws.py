"""Which labels of a Swendsen-Wang sweep take a second draw (plq_second_draws.h),
on the host against the sampler itself: labels drawn one after another from a
stream whose outputs ask for a second draw far more often than a real one's, so
that second draws follow each other and move labels past the listed places."""
import ctypes
import os
import random
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
HEADER = os.path.join(ROOT, "plaquette_b200", "csrc", "plq_second_draws.h")
CAP = 64


@pytest.fixture(scope="module")
def resolve(tmp_path_factory):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    d = tmp_path_factory.mktemp("second")
    (d / "resolve.cpp").write_text(
        f'#include "{HEADER}"\n'
        'extern "C" int resolve(int *place, int listed, long labels, const char *asks, int cap, int *rank) {\n'
        "    int n;\n"
        "    const bool ok = plq::resolve_second_draws(place, listed, labels, cap, rank, n,\n"
        "                                              [&](int64_t p) { return asks[p] != 0; });\n"
        "    return ok ? n : -1;\n}\n")
    subprocess.run([cxx, "-std=c++17", "-shared", "-fPIC", "-o", str(d / "resolve.so"), str(d / "resolve.cpp")], check=True)
    f = ctypes.CDLL(str(d / "resolve.so")).resolve
    f.argtypes = [ctypes.c_void_p, ctypes.c_int, ctypes.c_long, ctypes.c_char_p, ctypes.c_int, ctypes.c_void_p]

    def call(asks, labels, rng):
        listed = [p for p in range(labels) if asks[p]]
        rng.shuffle(listed)  # (the rank pass lists them in no order)
        place = (ctypes.c_int * max(1, len(listed)))(*listed)
        rank = (ctypes.c_int * CAP)()
        n = f(place, len(listed), labels, bytes(asks), CAP, rank)
        return None if n < 0 else list(rank[:n])

    return call


def sequential(asks, labels):
    p, out = 0, []
    for r in range(labels):
        if asks[p]:
            out.append(r)
            p += 1
        p += 1
    return out


@pytest.mark.parametrize("density", [0.0, 0.02, 0.2, 0.5, 1.0])
def test_ranks(resolve, density):
    rng = random.Random(7)
    for labels in list(range(1, 30)) + [100, 1000]:
        for _ in range(40):
            asks = [int(rng.random() < density) for _ in range(2 * labels + 2)]
            want = sequential(asks, labels)
            listed = sum(asks[:labels])
            assert resolve(asks, labels, rng) == (want if len(want) <= CAP and listed <= CAP else None)
