"""The swap search's work as its users call it: timed cases over the ranges the
framework declares, each through the public entry points of pyhea_b200.

    listed()             the cases, plain dicts
    draw(rng)            one more case of the same ranges
    prepare(case, seed)  what a program holds before the call (problems, plans, batches, a server)
    run(state)           one pass through the public entry points, its outputs as arrays
    work(case)           bytes and operations a pass cannot do without
    exact(case, seed)    float64 values of the computed outputs where they have one

Kinds of case (``case["kind"]``) and the real use behind them:

    recount   pair counts and fitness of given structures (``recount``): checking a written
              POSCAR (one structure, the smallest call) or a whole population
    generate  seeded random structures of a composition (``generate``)
    search    the whole search, host arrays in and out (``search``): one structure, one call
    dropin    the same through the pybind11 module as PyHEA calls it (nested lists in and out)
    plan      a kept plan run again with a new seed and read back (``Plan.run``, ``Plan.read``)
    batch     many structures of uneven size searched together (``Batch.run``, ``Batch.read``)
    serve     requests of mixed size submitted to a kept server and drained (``Server``)

Structures are the bench configurations of workloads.py at a few iterations: FCC
10^3 with 4 species, BCC 20^3 with 5, the mixed batch, FCC 100^3, the serving
mix; and the general ones around them: small cubes, supercells with three
different edges (their tables are no cube's), one to three shells, 2 to 6 species.
Sizes of a case are fixed by the case; compositions, targets, occupancies and
search seeds come from the seed given to ``prepare``.
"""
import math

import numpy as np

import pyhea_b200 as hb
from pyhea_b200 import lattice as L
from pyhea_b200 import workloads as W

_BASIS = {L.FCC: ((0, 0, 0), (1, 1, 0), (1, 0, 1), (0, 1, 1)), L.BCC: ((0, 0, 0), (1, 1, 1))}


def listed():
    return [
        # one structure's counts and fitness: the smallest call a user makes (checking one POSCAR)
        dict(name="recount_one", kind="recount", lat="fcc", x=6, y=6, z=6, types=4, shells=3, true3=False, count=1),
        # the counts of a saved population
        dict(name="recount_many", kind="recount", lat="bcc", x=24, y=24, z=24, types=5, shells=3, true3=False, count=64),
        # a population of random structures (the search's start, or a baseline for its result)
        dict(name="generate_many", kind="generate", lat="bcc", x=20, y=20, z=20, types=5, shells=3, true3=False,
             count=128, equal=True, amp=0.15),
        # PyHEA's own call on a small cell: nested lists in, nested lists out
        dict(name="dropin_small", kind="dropin", lat="bcc", x=6, y=6, z=6, types=3, shells=2, true3=False, P=16, Q=64,
             I=4, D=8),
        # one whole call of the CPU-sized configuration: FCC 10^3, 4 x 1000 atoms, 128 solutions x 256 tasks
        dict(name="search_fcc10", kind="search", lat="fcc", x=10, y=10, z=10, types=4, shells=3, true3=True, P=128,
             Q=256, I=10, D=10, equal=True, amp=0.1),
        # one whole call on a structure beyond shared memory, its 43 MB table given
        dict(name="search_fcc40", kind="search", lat="fcc", x=40, y=40, z=40, types=3, shells=3, true3=True, P=8,
             Q=1024, I=2, D=12, rounds=700),
        # a supercell with three different edges: a general table, six species
        dict(name="plan_box", kind="plan", lat="fcc", x=13, y=9, z=11, types=6, shells=3, true3=False, P=48, Q=200,
             I=6, D=12, rounds=0),
        # the headline configuration (BCC 20^3, 5 x 3200 atoms, 256 solutions x 512 tasks) for eight of its iterations
        dict(name="plan_bcc20", kind="plan", lat="bcc", x=20, y=20, z=20, types=5, shells=3, true3=False, P=256, Q=512,
             I=8, D=20, rounds=0, equal=True, amp=0.15),
        # structures of millions of sites: FCC 100^3, 32 solutions x 4096 tasks, searches capped at 1200 rounds
        dict(name="plan_fcc100", kind="plan", lat="fcc", x=100, y=100, z=100, types=4, shells=3, true3=True, P=32,
             Q=4096, I=1, D=20, rounds=1200, equal=True, amp=0.05),
        # a few small structures together: less work than the chip holds
        dict(name="batch_small", kind="batch", mix=3, count=12, low=4, high=9, P=24, Q=128, I=4, D=8),
        # the mixed batch: cells of edge 6 to 30, 64 solutions x 256 tasks
        dict(name="batch_mixed", kind="batch", mix=0, count=40, low=6, high=30, P=64, Q=256, I=3, D=10),
        # requests of 4e3 to 3e5 sites in one go, with the tolerance of the serving configuration
        dict(name="serve_mix", kind="serve", mix=1, count=10, n_min=4000, n_max=300000, P=16, Q=256, I=4, D=10,
             tol=1e-3),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _cell(rng, lo, hi, cube=None):
    """Lattice, edges and chemistry of one structure of lo..hi sites; a third of them no cubes."""
    lat = rng.choice(["fcc", "bcc"])
    nb = 4 if lat == "fcc" else 2
    edge = max(3, int(round((_log(rng, lo, hi) / nb) ** (1.0 / 3.0))))
    x = y = z = edge
    if cube is False or (cube is None and rng.random() < 0.33):
        x, y = edge + rng.randint(0, 2), max(3, edge - rng.randint(1, 2))
    return dict(lat=lat, x=x, y=y, z=z, types=rng.randint(2, 6), shells=rng.choice([1, 2, 3, 3, 3]),
                true3=lat == "fcc" and rng.random() < 0.6, equal=rng.random() < 0.4, amp=rng.choice([0.05, 0.1, 0.15]))


def draw(rng):
    kind = rng.choice(["recount", "generate", "dropin", "search", "search", "plan", "plan", "plan", "batch",
                       "batch", "serve"])
    if kind == "recount":
        c = _cell(rng, 400, 30000)
        return dict(kind=kind, **c, count=_log(rng, 1, 64))
    if kind == "generate":
        c = _cell(rng, 400, 30000)
        return dict(kind=kind, **c, count=_log(rng, 1, 128))
    if kind == "dropin":
        c = _cell(rng, 128, 1000)
        return dict(kind=kind, **c, P=rng.randint(4, 16), Q=_log(rng, 16, 128), I=rng.randint(1, 4),
                    D=rng.randint(4, 12))
    if kind == "search":
        c = _cell(rng, 400, 16000)
        return dict(kind=kind, **c, P=_log(rng, 8, 128), Q=_log(rng, 32, 512), I=rng.randint(1, 6),
                    D=rng.randint(4, 16))
    if kind == "plan":
        if rng.random() < 0.25:  # beyond shared memory: occupancies in HBM, capped searches
            c = _cell(rng, 260000, 2000000, cube=True)
            c["types"] = rng.randint(3, 5)
            return dict(kind=kind, **c, P=_log(rng, 8, 24), Q=_log(rng, 512, 4096), I=1, D=rng.randint(8, 20),
                        rounds=_log(rng, 200, 900))
        c = _cell(rng, 400, 24000)
        return dict(kind=kind, **c, P=_log(rng, 8, 192), Q=_log(rng, 32, 600), I=rng.randint(1, 6),
                    D=rng.randint(4, 20), rounds=0)
    if kind == "batch":
        low = rng.randint(4, 8)
        return dict(kind=kind, mix=rng.randint(10, 10**6), count=rng.randint(4, 32), low=low,
                    high=rng.randint(low + 2, 22), P=_log(rng, 8, 48), Q=_log(rng, 48, 256), I=rng.randint(1, 3),
                    D=rng.randint(4, 12))
    return dict(kind="serve", mix=rng.randint(10, 10**6), count=rng.randint(2, 10), n_min=2000,
                n_max=_log(rng, 8000, 120000), P=rng.randint(4, 16), Q=_log(rng, 64, 256), I=rng.randint(1, 4),
                D=rng.randint(4, 12), tol=rng.choice([-1.0, 1e-3]))


# ---- structures ----

def _lattice(case):
    return L.FCC if case["lat"] == "fcc" else L.BCC


def _shell_set(case):
    return L.SHELLS_FCC_TRUE3 if case["true3"] else L.SHELLS_REFERENCE


def _sites(case):
    return len(_BASIS[_lattice(case)]) * case["x"] * case["y"] * case["z"]


def _shell_sizes(case):
    return [len(v) for v in L.shell_vectors(_lattice(case), _shell_set(case))]


def _table(case):
    """Neighbour table [N][sum Z] of an x * y * z supercell, ids ascending within each shell (the
    numbering of lattice.py with the edges apart)."""
    basis = np.array(_BASIS[_lattice(case)])
    ex, ey, ez = case["x"], case["y"], case["z"]
    nb = len(basis)
    index = -np.ones(8, dtype=np.int64)
    for i, (a, b, c) in enumerate(basis):
        index[(a & 1) * 4 + (b & 1) * 2 + (c & 1)] = i
    s = np.arange(nb * ex * ey * ez)
    cell = s // nb
    pos = 2 * np.stack([cell // (ey * ez), (cell // ez) % ey, cell % ez], axis=1) + basis[s % nb]
    wrap = np.array([2 * ex, 2 * ey, 2 * ez])
    cols = []
    for vec in L.shell_vectors(_lattice(case), _shell_set(case)):
        q = (pos[:, None, :] + vec[None, :, :]) % wrap
        b = index[(q[..., 0] & 1) * 4 + (q[..., 1] & 1) * 2 + (q[..., 2] & 1)]
        cols.append(np.sort(nb * (((q[..., 0] >> 1) * ey + (q[..., 1] >> 1)) * ez + (q[..., 2] >> 1)) + b, axis=1))
    return np.concatenate(cols, axis=1).astype(np.int32)


def _chemistry(case, rng):
    """Composition, target and weights of one structure: (nearly) equal counts with the plain
    configurations' target, or the batched configuration's Dirichlet(2) counts and projected target."""
    n, t, s, amp = _sites(case), case["types"], case["shells"], case.get("amp", 0.1)
    if case.get("equal"):
        species = np.full(t, n // t, dtype=np.int32)
        species[: n % t] += 1
        return species, W.zero_row_sum_target(rng, t, amp, shells=s), W.WEIGHTS[:s]
    species = W.dirichlet_counts(rng, t, n)
    return species, W.projected_target(rng, species / n, amp, shells=s), W.WEIGHTS[:s]


def _problem(case, rng):
    species, target, weight = _chemistry(case, rng)
    if case["x"] == case["y"] == case["z"]:
        table, _ = hb.build_neighbors(_lattice(case), case["x"], _shell_set(case))
    else:
        table = _table(case)
    return hb.Problem(table, _shell_sizes(case), species, weight, target)


def _population(case, rng, species):
    one = np.repeat(np.arange(len(species), dtype=np.uint8), species)
    return np.stack([rng.permutation(one) for _ in range(case["count"])])


def _members(case):
    """Lattice, edge and species count of each structure of a batch, fixed by the case."""
    rng = np.random.default_rng(case["mix"])
    return [(int(rng.integers(0, 2)), int(rng.integers(case["low"], case["high"] + 1)), int(rng.integers(3, 7)))
            for _ in range(case["count"])]


def _requests(case):
    """Lattice, edge and species count of each request: site counts spread over their logarithm."""
    rng = np.random.default_rng(case["mix"])
    out = []
    for _ in range(case["count"]):
        lat = int(rng.integers(0, 2))
        nb = 4 if lat == L.FCC else 2
        n = math.exp(rng.uniform(math.log(case["n_min"]), math.log(case["n_max"])))
        out.append((lat, max(4, int(round((n / nb) ** (1.0 / 3.0)))), int(rng.integers(3, 7))))
    return out


# ---- the pass ----

def prepare(case, seed):
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    state = dict(case=case, seed=int(rng.integers(1, 2**62)))
    if kind in ("recount", "generate", "search"):
        state["problem"] = _problem(case, rng)
        if kind == "recount":
            state["occ"] = _population(case, rng, state["problem"].species)
    elif kind == "dropin":
        species, target, weight = _chemistry(case, rng)
        state["args"] = (L.as_nested(_table(case), _shell_sizes(case)), [int(v) for v in species], list(weight),
                         [list(row) for row in target])
        hb.accelerate.cuda_available()
    elif kind == "plan":
        cube = case["x"] == case["y"] == case["z"]
        if cube and _sites(case) > 200000:  # no table: a lattice description
            species, target, weight = _chemistry(case, rng)
            problem = hb.Problem.from_lattice(_lattice(case), case["x"], species, weight, target,
                                              shell_set=_shell_set(case))
        else:
            problem = _problem(case, rng)
        state["plan"] = hb.Plan(problem, case["P"], case["I"], case["Q"], case["D"], max_rounds=case["rounds"])
    elif kind == "batch":
        problems, params = [], []
        for lat, edge, types in _members(case):
            species = W.dirichlet_counts(rng, types, L.num_sites(lat, edge))
            target = W.projected_target(rng, species / species.sum(), 0.1)
            shell_set = L.SHELLS_FCC_TRUE3 if lat == L.FCC else L.SHELLS_REFERENCE
            problems.append(hb.Problem.from_lattice(lat, edge, species, W.WEIGHTS, target, shell_set=shell_set))
            params.append(dict(num_solutions=case["P"], total_iter=case["I"], parallel_task=case["Q"],
                               converge_depth=case["D"]))
        state["batch"] = hb.Batch(problems, params)
        state["seeds"] = [int(v) for v in rng.integers(1, 2**62, size=case["count"])]
    elif kind == "serve":
        state["server"] = hb.Server(arena_bytes=4 << 30)
        state["requests"] = []
        for i, (lat, edge, types) in enumerate(_requests(case)):
            species = W.dirichlet_counts(rng, types, L.num_sites(lat, edge))
            target = W.projected_target(rng, species / species.sum(), 0.1)
            shell_set = L.SHELLS_FCC_TRUE3 if lat == L.FCC else L.SHELLS_REFERENCE
            state["requests"].append((lat, edge, species, target, shell_set,
                                      dict(num_solutions=case["P"], total_iter=case["I"], parallel_task=case["Q"],
                                           converge_depth=case["D"], seed=int(rng.integers(1, 2**62)))))
    return state


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "recount":
        return hb.recount(state["problem"], state["occ"])
    if kind == "generate":
        return hb.generate(state["problem"], state["seed"], 0, case["count"])
    if kind == "search":
        occ, fit, stats = hb.search(state["problem"], case["P"], case["I"], case["Q"], case["D"], seed=state["seed"],
                                    max_rounds=case.get("rounds", 0))
        return occ, fit, stats["evals"]
    if kind == "dropin":
        nbor, species, weight, target = state["args"]
        rows, fit = hb.accelerate.run_local_parallel_hcs_cuda(case["P"], case["I"], case["Q"], case["D"], 0.001, nbor,
                                                              species, weight, target, seed=state["seed"],
                                                              verbose=False)
        return np.array(rows, dtype=np.uint8), np.array(fit)
    if kind == "plan":
        stats = state["plan"].run(state["seed"])
        occ, fit = state["plan"].read()
        return occ, fit, stats["evals"]
    if kind == "batch":
        batch = state["batch"]
        stats = batch.run(state["seeds"])
        results = [batch.read(i) for i in range(case["count"])]
        return [r[0] for r in results], np.concatenate([r[1] for r in results]), stats["evals"]
    server = state["server"]
    ids = [server.submit_lattice(lat, edge, species, W.WEIGHTS, target, params, shell_set=shell_set,
                                 tolerance=case["tol"])
           for lat, edge, species, target, shell_set, params in state["requests"]]
    server.drain()
    server.take_finished()
    results = [server.result(i) for i in ids]
    return ([r[0] for r in results], np.concatenate([r[1] for r in results]),
            np.array([r[2]["iterations"] for r in results]), np.array([r[2]["evals"] for r in results]))


# ---- what a pass cannot do without ----

def _search_work(n, z, types, shells, P, Q, I, D, rounds=0, reach=0.45):
    """Bytes and operations of one structure's search.  Per local search from a random structure:
    about reach * n^(2/3) (512 / Q)^(1/4) rounds of Q proposals (the measured trend; `reach` grows with
    how far the target is from random), at least D; per survivors' search at least D rounds.  A
    proposal needs both sites' neighbourhood counts (one 16-byte entry each) and a fused multiply-add
    pair for each species and shell; a new structure its n species written and its n * z neighbours
    counted."""
    long = max(D, reach * n ** (2.0 / 3.0) * (512.0 / Q) ** 0.25)
    if rounds:
        long, D = min(long, rounds), min(rounds, D)
    evals = I * P * Q * (long + D)
    new = (I + 1) * P * n
    return dict(bytes=32.0 * evals + 17.0 * new + P * n, flops=4.0 * shells * (types + 1) * evals + new * z)


def work(case):
    kind = case["kind"]
    if kind in ("batch", "serve"):
        members = _members(case) if kind == "batch" else _requests(case)
        I = case["I"] if kind == "batch" else 1  # a request may reach its tolerance in one iteration
        parts = [_search_work(L.num_sites(lat, edge), 42 if lat == L.FCC else 26, types, 3, case["P"], case["Q"], I,
                              case["D"]) for lat, edge, types in members]
    else:
        n, z = _sites(case), sum(_shell_sizes(case)[: case["shells"]])
        if kind in ("recount", "generate"):
            out = n + 4.0 * case["types"] ** 2 * case["shells"] + 8
            return dict(bytes=4.0 * n * z + case["count"] * out, flops=float(case["count"]) * n * z)
        reach = (8.0 if case.get("equal") else 4.5) * case.get("amp", 0.1)
        parts = [_search_work(n, z, case["types"], case["shells"], case["P"], case["Q"], case["I"], case["D"],
                              case.get("rounds", 0), reach)]
    return dict(bytes=sum(p["bytes"] for p in parts), flops=sum(p["flops"] for p in parts))


def exact(case, seed):
    """Recounts have their values in closed form; a search's outputs are the result of a seeded
    sequence of choices (whole numbers, compared as such), so they have none."""
    if case["kind"] != "recount":
        return None
    rng = np.random.default_rng(seed)
    rng.integers(1, 2**62)
    species, target, weight = _chemistry(case, rng)
    table, sizes, t, n = _table(case), _shell_sizes(case), case["types"], _sites(case)
    occ = _population(case, rng, species).astype(np.int64)
    c = species.astype(np.float64) / n
    counts = np.empty((len(occ), case["shells"], t, t), dtype=np.int32)
    f2 = np.zeros(len(occ))
    for p, row in enumerate(occ):
        off = 0
        for k in range(case["shells"]):
            pair = row[:, None] * t + row[table[:, off:off + sizes[k]]]
            counts[p, k] = np.bincount(pair.ravel(), minlength=t * t).reshape(t, t)
            off += sizes[k]
            alpha = 1.0 - counts[p, k] / (sizes[k] * float(n)) / np.outer(c, c)
            f2[p] += weight[k] * np.sum((alpha - target[k].reshape(t, t)) ** 2)
    return counts, f2
