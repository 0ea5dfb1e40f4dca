"""The hand-shake of a Wolff launch (wolff_kernel in plq_cluster.cu), explored on
the host: every interleaving of the growing CTA and the waiting ones over short
runs of updates -- small ones that call no one (u), called ones whose cluster the
growth finds whole (w), large ones (L) -- with the kernel's own decision function.
All CTAs have to leave each barrier from the same place, take the right branch
after it, and reach the end."""
import ctypes
import itertools
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
HEADER = os.path.join(ROOT, "plaquette_b200", "csrc", "plq_wolff_sync.h")


@pytest.fixture(scope="module")
def ended(tmp_path_factory):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    d = tmp_path_factory.mktemp("wolff")
    (d / "ended.cpp").write_text(
        f'#include "{HEADER}"\n'
        'extern "C" int ended(unsigned long long word, unsigned long long id) {\n'
        "    return plq::wolff_ended_by_growth(word, id);\n}\n")
    subprocess.run([cxx, "-shared", "-fPIC", "-o", str(d / "ended.so"), str(d / "ended.cpp")], check=True)
    f = ctypes.CDLL(str(d / "ended.so")).ended
    f.argtypes = [ctypes.c_ulonglong] * 2
    table = {(w, i): bool(f(w, i)) for w in range(10) for i in range(10)}
    return lambda word, i: table[word, i]


def explore(outcomes, ctas, ended):
    """All interleavings; a CTA is (step, update, barrier of the update), the memory (call, small0, small1)."""
    last = len(outcomes) + 1

    def step(cta, who, call, small):
        """The CTA's next states and memory; None while it waits."""
        at, i, b = cta
        if who == 0 and at == "next":  # the growing CTA goes on to update i + 1
            i += 1
            if i == last:
                return ("done", i, 0), last, small
            if outcomes[i - 1] == "u":
                return ("next", i, 0), call, small
            return ("mark", i, 0), i, small
        if at == "mark":
            if outcomes[i - 1] == "w":
                small = (i, small[1]) if i % 2 == 0 else (small[0], i)
            return ("arrive", i, 0), call, small
        if at == "next":  # a waiting CTA
            if call <= i:
                return None
            return (("done", call, 0) if call == last else ("arrive", call, 0)), call, small
        if at == "arrive":
            return ("wait", i, b), call, small
        if at == "read":
            stop = ended(small[i % 2], i)
            assert stop == (outcomes[i - 1] == "w"), (outcomes, i, who)
            return (("next", i, 0) if stop else ("arrive", i, 1)), call, small
        return None  # wait, done

    start = ((("next", 0, 0),) * ctas, 0, (0, 0))
    seen, todo = {start}, [start]
    while todo:
        state, call, small = todo.pop()
        if all(c[0] == "done" for c in state):
            continue
        if all(c[0] == "wait" for c in state):  # the barrier opens
            assert len(set(state)) == 1, (outcomes, state)
            _, i, b = state[0]
            after = [((("read", i, 0) if b == 0 else ("arrive", i, 2) if b == 1 else ("next", i, 0)),) * ctas]
            following = [(after[0], call, small)]
        else:
            following = []
            for who, cta in enumerate(state):
                moved = step(cta, who, call, small)
                if moved:
                    following.append((state[:who] + (moved[0],) + state[who + 1:], moved[1], moved[2]))
            assert following, ("stuck", outcomes, state)
        for s in following:
            if s not in seen:
                seen.add(s)
                todo.append(s)


@pytest.mark.parametrize("ctas", [2, 3])
def test_every_interleaving(ended, ctas):
    for outcomes in itertools.product("uwL", repeat=5):
        explore(outcomes, ctas, ended)
