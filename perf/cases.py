"""The work that users of this framework have it do, as cases that can be timed.

A case is a dict of plain values.  ``listed()`` names twelve of them, ``draw(rng)``
gives further ones of the same ranges, ``prepare`` builds what a program has in
hand before its call (a chain, an ensemble or a server on the device, from a
seeded start), ``run`` is one pass through the public entry points, and ``work``
counts what that pass cannot do without.  Five kinds:

* ``chain``    -- a local-update chain (Ising, Potts or Z2 gauge; Metropolis or
  heat bath; PCG or keyed stream): ``samples`` samples, ``sweeps`` sweeps apart,
  with their primaries, and either every configuration or the last one; then
  the correlator or the loops, where the case measures them.
* ``sw``       -- Swendsen-Wang sweeps, a sample and the cluster-size histogram.
* ``wolff``    -- single-cluster updates, then a sample.
* ``ensemble`` -- 4D gauge lattices beside 3D Ising tempering ladders, blocks of
  sweeps with every member's primaries and betas, then every configuration.
* ``serve``    -- a burst of mixed jobs, submitted at once and waited for.

All outputs are whole numbers (the ensemble's betas are copies of its inputs),
so ``exact`` has nothing to add.
"""
import numpy as np

import plaquette_b200 as plq
from plaquette_b200.ensemble import build_ensemble
from plaquette_b200.serving import JOB_DONE, Server, random_job

MODELS = {"ising": plq.ISING, "potts": plq.POTTS, "gauge": plq.GAUGE}
UPDATERS = {"metropolis": plq.METROPOLIS, "heatbath": plq.HEATBATH}
STREAMS = {"pcg": plq.RNG_STREAM, "keyed": plq.RNG_KEYED}

# Couplings near the transition, where these chains are run in earnest.
BETA_C = {("ising", 2, 2): 0.4406868, ("ising", 2, 3): 0.2216544, ("ising", 2, 4): 0.1496947,
          ("gauge", 2, 3): 0.7614, ("gauge", 2, 4): 0.4407,
          ("potts", 2, 2): 0.8813736, ("potts", 3, 2): 1.0050525, ("potts", 4, 2): 1.0986123,
          ("potts", 5, 2): 1.1743590, ("potts", 6, 2): 1.2382, ("potts", 7, 2): 1.2935,
          ("potts", 2, 3): 0.4433088, ("potts", 3, 3): 0.5505, ("potts", 4, 3): 0.6286, ("potts", 5, 3): 0.69,
          ("potts", 6, 3): 0.74, ("potts", 7, 3): 0.78}

# Integer operations of one draw: two lowbias32 rounds; a 128-bit LCG step with its output function.
KEYED_OPS, PCG_OPS = 18, 30


def chain_case(model, q, shape, updater, stream, sweeps, samples, states=False, measure="none", name=None):
    c = {"kind": "chain", "model": model, "q": q, "shape": shape, "updater": updater, "stream": stream,
         "sweeps": sweeps, "samples": samples, "states": states, "measure": measure}
    return dict(c, name=name) if name else c


def cluster_case(kind, model, q, shape, stream, updates, name=None):
    c = {"kind": kind, "model": model, "q": q, "shape": shape, "stream": stream, "updates": updates}
    return dict(c, name=name) if name else c


def listed():
    return [
        # the textbook run: a small critical 2D lattice, energy and magnetisation every 10 sweeps
        chain_case("ising", 2, "64x64", "metropolis", "pcg", 10, 100, name="ising-64x64-series"),
        # a small uneven 3D lattice whose every configuration is kept: launches and latency count
        chain_case("ising", 2, "48x40x36", "heatbath", "keyed", 5, 20, states=True, name="ising-48x40x36-samples"),
        # the largest lattice on the keyed stream, energies now and then
        chain_case("ising", 2, "512x512x512", "metropolis", "keyed", 100, 8, name="ising-512-keyed"),
        # the largest Potts run, bit-exact stream, order parameter every 10 sweeps
        chain_case("potts", 3, "512x512x512", "heatbath", "pcg", 10, 30, name="potts3-512-pcg"),
        # a mid-size lattice on the bit-exact stream with its correlation function
        chain_case("ising", 2, "256x256x256", "metropolis", "pcg", 20, 10, measure="correlator",
                   name="ising-256-pcg-correlator"),
        # one 4D gauge lattice, Wilson and Polyakov loops after its sweeps
        chain_case("gauge", 2, "24x24x24x24", "heatbath", "keyed", 10, 10, measure="loops", name="gauge-24-loops"),
        # many-state Potts on an uneven lattice
        chain_case("potts", 5, "1002x750", "metropolis", "keyed", 20, 5, name="potts5-1002x750"),
        # critical slowing down avoided: Swendsen-Wang on a large 2D lattice
        cluster_case("sw", "ising", 2, "4096x4096", "keyed", 100, name="sw-4096"),
        # Swendsen-Wang, 3D Potts, bit-exact stream
        cluster_case("sw", "potts", 3, "96x96x96", "pcg", 50, name="sw-potts3-96-pcg"),
        # Wolff updates of a critical 3D lattice
        cluster_case("wolff", "ising", 2, "128x128x128", "keyed", 500, name="wolff-128"),
        # replicas: 64 gauge lattices beside five tempering ladders of 256 Ising lattices
        {"kind": "ensemble", "gauge": "8,12,16,24", "gauge_each": 16, "ising": "16,24,32,48,64",
         "ladders": "52,51,51,51,51", "sweeps": 100, "blocks": 3, "name": "ensemble"},
        # a burst of mixed jobs on the serving loop
        {"kind": "serve", "jobs": 24, "mix": 11, "scale": 0.1, "name": "serve-burst"},
    ]


# ------------------------------------------------------------------ draw
def _log(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def _even(rng, lo, hi):
    return max(2, 2 * (_log(rng, lo, hi) // 2))


def _extents(rng, d, lo, hi):
    """Even extents, log-uniform; half of the shapes uneven, some with a first extent that suits vectors."""
    L = _even(rng, lo, hi)
    ext = [L] * d
    if rng.random() < 0.5:
        ext = [max(2, 2 * int(L * rng.uniform(0.7, 1.3) / 2)) for _ in range(d)]
    if L >= 64 and rng.random() < 0.5:
        ext[0] = 64 * max(1, ext[0] // 64)
    return ext


def _volume(ext):
    n = 1
    for L in ext:
        n *= L
    return n


def _text(ext):
    return "x".join(str(L) for L in ext)


def draw(rng):
    kind = rng.choice(["sites", "sites", "sites", "gauge", "gauge", "sw", "sw", "wolff", "ensemble", "serve"])
    if kind == "sites":
        d = rng.choice([2, 2, 3, 3])
        ext = _extents(rng, d, 16, 4096) if d == 2 else _extents(rng, d, 8, 400)
        q = rng.choice([2, 2, 3, 4, 5])
        model = "ising" if q == 2 and rng.random() < 0.7 else "potts"
        updater = rng.choice(["metropolis", "heatbath"])
        # (Metropolis proposals at q > 2 on the bit-exact stream are one sequential walk)
        stream = rng.choice(["pcg", "keyed"]) if q == 2 or updater == "heatbath" else "keyed"
        n = _volume(ext)
        sweeps = rng.choice([1, 5, 10, 20])
        samples = max(1, min(100, int(6e9 / (n * sweeps))))
        states = n * samples < 2e7 and rng.random() < 0.5
        measure = "correlator" if rng.random() < 0.25 else "none"
        return chain_case(model, q, _text(ext), updater, stream, sweeps, samples, states, measure)
    if kind == "gauge":
        d = rng.choice([3, 4])
        ext = _extents(rng, d, 4, 96) if d == 3 else _extents(rng, d, 4, 32)
        n = _volume(ext) * d
        sweeps = rng.choice([1, 5, 10])
        samples = max(1, min(40, int(4e8 / (n * sweeps))))
        states = n * samples < 2e7 and rng.random() < 0.5
        measure = "loops" if rng.random() < 0.4 else "none"
        return chain_case("gauge", 2, _text(ext), rng.choice(["metropolis", "heatbath"]),
                          rng.choice(["pcg", "keyed"]), sweeps, samples, states, measure)
    if kind in ("sw", "wolff"):
        d = rng.choice([2, 3])
        hi = 4096 if kind == "sw" else 1024
        ext = _extents(rng, d, 32, hi) if d == 2 else _extents(rng, d, 12, 160 if kind == "sw" else 128)
        q = rng.choice([2, 2, 3, 4])
        model = "ising" if q == 2 else "potts"
        n = _volume(ext)
        if kind == "sw":
            updates = max(2, min(100, int(1.5e9 / n)))
            return cluster_case("sw", model, q, _text(ext), rng.choice(["pcg", "keyed"]), updates)
        return cluster_case("wolff", model, q, _text(ext), "keyed", _log(rng, 50, 500))
    if kind == "ensemble":
        gauge = sorted(rng.sample([4, 6, 8, 10, 12, 14, 16, 18, 20], rng.randint(1, 3)))
        ising = sorted(rng.sample([8, 12, 16, 20, 24, 28, 32, 40, 48, 56], rng.randint(1, 4)))
        return {"kind": "ensemble", "gauge": ",".join(map(str, gauge)), "gauge_each": rng.randint(2, 16),
                "ising": ",".join(map(str, ising)), "ladders": ",".join(str(rng.randint(4, 40)) for _ in ising),
                "sweeps": 10 * rng.randint(1, 10), "blocks": rng.randint(1, 3)}
    return {"kind": "serve", "jobs": rng.randint(4, 24), "mix": rng.randint(1, 10 ** 6),
            "scale": round(rng.uniform(0.02, 0.06), 3)}


# --------------------------------------------------------------- prepare
def _shape(case):
    return tuple(int(t) for t in case["shape"].split("x"))


def _n_vars(case):
    shape = _shape(case)
    return _volume(shape) * (len(shape) if case["model"] == "gauge" else 1)


def _start(case, seed):
    return np.random.default_rng(seed).integers(0, case["q"], size=_n_vars(case), dtype=np.uint8)


def _beta(case):
    return BETA_C[(case["model"], case["q"], len(_shape(case)))]


_gpu = None


def _device():
    global _gpu
    if _gpu is None:
        _gpu = plq.Gpu.new()
    return _gpu


def _prepare_chain(case, seed):
    desc = plq.make_desc(MODELS[case["model"]], case["q"], _shape(case), UPDATERS[case["updater"]],
                         beta=_beta(case), seed=seed, rng=STREAMS[case["stream"]], sweeps_between=case["sweeps"],
                         batch=case["samples"])
    chain = plq.GpuChain(_device(), desc, _start(case, seed))
    chain.advance(10)  # off the random start
    chain.sync()
    return chain


def _cluster_chain(case, seed, start, kind, stream, sweeps):
    make = plq.GpuClusterChain.swendsen_wang if kind == "sw" else plq.GpuClusterChain.wolff
    return make(_device(), _shape(case), MODELS[case["model"]], case["q"], 1.0, _beta(case), seed, start, sweeps,
                rng=STREAMS[stream])


def _prepare_cluster(case, seed):
    # clusters have their critical sizes only near equilibrium: Swendsen-Wang sweeps first
    warm = _cluster_chain(case, seed, _start(case, seed), "sw", "keyed", 1)
    warm.advance(40)
    start = warm.read()
    warm.close()
    return _cluster_chain(case, seed + 1, start, case["kind"], case["stream"], case["updates"])


def _numbers(text):
    return [int(t) for t in text.split(",")]


def _prepare_ensemble(case, seed):
    rng = np.random.default_rng(seed)
    descs, starts, ladders = [], [], []

    def add(desc, n):
        descs.append(desc)
        starts.append(rng.integers(0, 2, size=n, dtype=np.uint8))

    for L in _numbers(case["gauge"]):
        for beta in np.linspace(0.40, 0.48, case["gauge_each"]):
            add(plq.make_desc(plq.GAUGE, 2, (L,) * 4, plq.HEATBATH, beta=float(beta), seed=seed + len(descs),
                              rng=plq.RNG_KEYED, batch=1), 4 * L ** 4)
    for L, k in zip(_numbers(case["ising"]), _numbers(case["ladders"])):
        betas = [float(b) for b in np.geomspace(0.20, 0.24, k)]
        ladders.append((list(range(len(descs), len(descs) + k)), betas))
        for beta in betas:
            add(plq.make_desc(plq.ISING, 2, (L,) * 3, plq.METROPOLIS, beta=beta, seed=seed + len(descs),
                              rng=plq.RNG_KEYED, batch=1), L ** 3)
    return build_ensemble(_device(), descs, starts, ladders, seed=seed)


def _jobs(case, seed):
    """The case's jobs: descriptors of the serving mix, each with its own seed."""
    rng = np.random.default_rng(case["mix"])
    jobs = []
    for i in range(case["jobs"]):
        desc, sweeps = random_job(rng, seed * 1000 + i)
        jobs.append((desc, max(1, int(sweeps * case["scale"]))))
    return jobs


def prepare(case, seed):
    kind = case["kind"]
    if kind == "chain":
        return case, _prepare_chain(case, seed)
    if kind in ("sw", "wolff"):
        return case, _prepare_cluster(case, seed)
    if kind == "ensemble":
        return case, _prepare_ensemble(case, seed)
    return case, (Server(_device(), max_slots=64), _jobs(case, seed))


# ------------------------------------------------------------------- run
def run(state):
    case, held = state
    kind = case["kind"]
    if kind == "chain":
        states, primaries = held.next_batch(case["samples"], states=case["states"])
        out = {"primaries": primaries, "states": states if case["states"] else held.read()}
        if case["measure"] == "correlator":
            out["correlator"] = np.concatenate(held.axis_pair_sums())
        elif case["measure"] == "loops":
            out["wilson"], _ = held.wilson(6)
            out["polyakov"] = held.polyakov(len(_shape(case)) - 1)[0]
        return out
    if kind == "sw":
        states, primaries = held.next_sample()
        return {"states": states, "primaries": primaries, "sizes": held.size_histogram()}
    if kind == "wolff":
        states, primaries = held.next_sample()
        return {"states": states, "primaries": primaries}
    if kind == "ensemble":
        series, betas = [], []
        for _ in range(case["blocks"]):
            held.advance(case["sweeps"])
            series.append(np.concatenate(held.primaries_all()))
            betas.append(held.betas())
        return {"primaries": np.stack(series), "betas": np.stack(betas),
                "states": np.concatenate([held.read(m) for m in range(held.n)])}
    server, jobs = held
    ids = [server.submit(desc, None, sweeps, want_states=True) for desc, sweeps in jobs]
    out = []
    for job in ids:
        if server.wait(job) != JOB_DONE:
            raise RuntimeError("job %d did not finish" % job)
        states, primaries, _ = server.result(job, states=True)
        server.release(job)
        out += [states, primaries]
    return {"states": np.concatenate(out[0::2]), "primaries": np.concatenate(out[1::2])}


# ------------------------------------------------------------------ work
def work(case):
    """Bytes: each configuration that goes in or comes out once (one byte a variable, as
    they are kept), the correlator and the loops one more read.  Operations: the integer
    operations of the draws that the updates are defined by."""
    kind = case["kind"]
    if kind == "chain":
        n = _n_vars(case)
        updates = n * case["sweeps"] * case["samples"]
        out = case["samples"] if case["states"] else 1
        ops = KEYED_OPS if case["stream"] == "keyed" else PCG_OPS
        if case["updater"] == "metropolis" and (case["q"] > 2 or case["stream"] == "pcg"):
            ops *= 1.5 if case["q"] > 2 else 0.7  # a proposal besides; draws of uphill moves only
        return {"bytes": n * (1 + out + (case["measure"] != "none")), "flops": updates * ops}
    if kind in ("sw", "wolff"):
        n, d = _n_vars(case), len(_shape(case))
        ops = KEYED_OPS if case["stream"] == "keyed" else PCG_OPS
        if kind == "sw":
            return {"bytes": 2 * n, "flops": case["updates"] * n * d * ops}
        cluster = n ** (0.875 if d == 2 else 0.655)  # sites of a critical cluster
        return {"bytes": 2 * n, "flops": case["updates"] * cluster * d * ops}
    if kind == "ensemble":
        n = sum(4 * L ** 4 * case["gauge_each"] for L in _numbers(case["gauge"]))
        n += sum(L ** 3 * k for L, k in zip(_numbers(case["ising"]), _numbers(case["ladders"])))
        return {"bytes": 2 * n, "flops": n * case["sweeps"] * case["blocks"] * KEYED_OPS}
    n = updates = 0
    for desc, sweeps in _jobs(case, 0):
        v = int(np.prod([desc.shape[i] for i in range(desc.d)])) * (desc.d if desc.model == plq.GAUGE else 1)
        n += v
        updates += v * sweeps
    return {"bytes": n, "flops": updates * KEYED_OPS}


def exact(case, seed):
    return None
