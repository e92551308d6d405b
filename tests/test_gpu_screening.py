"""Proposals are screened in FP32 and decided exactly: whole searches equal the
oracle bit for bit where the screening's choices are hardest -- many equal D's
(two species, one shell), a species of a single atom, targets already met,
weights or targets outside FP32's range, six species in three shells (both
histogram widths) -- and where a round takes several passes (CTAs smaller than
the round, on one CTA and on a cluster, in both draw modes), with and without
the screening."""
from fractions import Fraction

import numpy as np
import pytest

import pyhea_b200 as hb
from oracle import hea_oracle as ho
from pyhea_b200 import lattice as L
from pyhea_b200 import workloads as W

pytestmark = pytest.mark.gpu


def problems(lattice, cell, species, shells, shell_set=L.SHELLS_REFERENCE, seed=0, weight=None, scale=1.0, recognize=True):
    st = W.small_case(lattice=lattice, cell=cell, species=species, shells=shells, shell_set=shell_set, seed=seed)
    nbor, sizes = st.neighbors()
    weight = st.weight if weight is None else weight
    target = scale * np.asarray(st.target)
    row = int(sizes[:shells].sum())
    return (hb.Problem(nbor, sizes, st.species, weight, target, recognize=recognize),
            ho.Problem(nbor[:, :row], sizes[:shells], st.species, weight, target))


def same(gp, op, P, I, Q, D, seed, **kw):
    occ, fit, stats = hb.search(gp, P, I, Q, D, seed=seed, **kw)
    kw.pop("hbm_occupancy", None)
    wocc, wf2, wstats = op.hcs(seed, P, I, Q, D, **kw)
    np.testing.assert_array_equal(occ, wocc)
    np.testing.assert_array_equal(fit, np.sqrt(wf2))
    assert (stats["evals"], stats["accepts"], stats["rounds"]) == (wstats["evals"], wstats["accepts"], wstats["rounds"])


@pytest.mark.parametrize("species,shells,weight,scale", [
    ((128, 128), 1, None, 1.0),            # few distinct D's: ties in every round
    ((255, 1), 2, None, 1.0),              # one atom of a species
    ((100, 100, 55, 1), 3, None, 1.0),
    ((86, 85, 85), 3, None, 0.0),          # target of random structures: D near 0
    ((64, 64, 64, 64), 3, [1e-40, 1e-41, 1e-42], 1.0),
    ((64, 64, 64, 64), 3, [1e30, 1.0, 1e-30], 1.0),
    ((64, 64, 64, 64), 3, [1e-300, 1.0, 1e300], 1.0),  # beyond FP32's range: every proposal exact
    ((64, 64, 64, 64), 3, [0.0, 1.0, 0.0], 1.0),
    ((64, 64, 64, 64), 3, [0.0, 0.0, 0.0], 1.0),
    ((64, 64, 64, 64), 3, None, 1e9),      # targets far outside
])
@pytest.mark.parametrize("hbm", [False, True])
def test_hard_choices(species, shells, weight, scale, hbm):
    gp, op = problems(L.FCC, 4, species, shells, seed=len(species), weight=weight, scale=scale)
    same(gp, op, 3, 2, 96, 3, seed=77, max_rounds=150, hbm_occupancy=hbm)


@pytest.mark.parametrize("lattice,shell_set", [(L.FCC, L.SHELLS_FCC_TRUE3), (L.FCC, L.SHELLS_REFERENCE), (L.BCC, 0)])
@pytest.mark.parametrize("recognize", [True, False])
@pytest.mark.parametrize("hbm", [False, True])
def test_six_species(lattice, shell_set, recognize, hbm):
    n = L.num_sites(lattice, 5)
    species = W.dirichlet_counts(np.random.default_rng(6), 6, n)
    gp, op = problems(lattice, 5, species, 3, shell_set, seed=2, recognize=recognize)
    same(gp, op, 3, 2, 200, 4, seed=9, hbm_occupancy=hbm)


@pytest.mark.parametrize("tasks", [257, 400, 512, 600, 769])
def test_passes_of_small_ctas(tasks):
    """More solutions in flight than one CTA of 512 threads per SM pair: CTAs of at most 256 threads."""
    gp, op = problems(L.BCC, 3, (20, 17, 17), 2, seed=tasks)
    same(gp, op, 75, 8, tasks, 2, seed=tasks)


@pytest.mark.parametrize("cell,tasks", [(6, 9000), (27, 8200), (27, 4097)])
def test_passes_on_a_cluster(cell, tasks):
    n = L.num_sites(L.FCC, cell)
    gp, op = problems(L.FCC, cell, [n // 4] * 4, 3, L.SHELLS_FCC_TRUE3, seed=1)
    same(gp, op, 2, 1, tasks, 3, seed=5, max_rounds=25, hbm_occupancy=True)


OUTSIDE = [
    ((64, 64, 64, 64), 3, [1e-300, 1.0, 1e300], 1.0),
    ((64, 64, 64, 64), 3, None, 1e9),
    ((100, 100, 55, 1), 2, None, 1e8),
    ((128, 128), 1, None, 1e9),
    ((60, 50, 50, 40, 30, 26), 3, [1e-300, 1.0, 1e300], 1.0),
]


@pytest.mark.parametrize("species,shells,weight,scale", OUTSIDE)
@pytest.mark.parametrize("tasks,hbm", [(513, False), (600, False), (1100, False), (4200, True), (8200, True)])
def test_passes_with_every_proposal_exact(species, shells, weight, scale, tasks, hbm):
    """Beyond FP32's range no interval tells an empty record from a proposal: passes after one that
    improved nothing (most of a survivors' search), on one CTA and on clusters, to convergence or
    some rounds past it."""
    gp, op = problems(L.FCC, 4, species, shells, seed=len(species), weight=weight, scale=scale)
    same(gp, op, 2, 2, tasks, 4, seed=tasks, max_rounds=40 if tasks > 2000 else 150, hbm_occupancy=hbm)


@pytest.mark.parametrize("species,shells,weight,scale", OUTSIDE)
def test_batch_passes_with_every_proposal_exact(species, shells, weight, scale):
    cases = [problems(L.FCC, 4, species, shells, seed=i, weight=weight, scale=scale) for i in range(3)]
    tasks = (257, 300, 700)
    b = hb.Batch([gp for gp, _ in cases],
                 [dict(num_solutions=3, total_iter=2, parallel_task=t, converge_depth=4, max_rounds=150) for t in tasks])
    for seeds in ((5, 6, 7), (8, 9, 10)):
        b.run(seeds)
        for i, (_, op) in enumerate(cases):
            wocc, wf2, _ = op.hcs(seeds[i], 3, 2, tasks[i], 4, max_rounds=150)
            occ, fit = b.read(i)[:2]
            np.testing.assert_array_equal(occ, wocc)
            np.testing.assert_array_equal(fit, np.sqrt(wf2))
    b.close()


def fma(a, b, c):
    return float(Fraction(a) * Fraction(b) + Fraction(c))


def asymmetric_target(op, C, rng, x):
    """Two species, one shell: targets with 1 - target = C R +- x off the diagonal (about), such that the swap
    with u = (1, -1) has D < 0 by the rounding of d_01 + d_10 alone (about 2^-53 x), while the sums rounded once
    put D above zero by more than the screening's bound."""
    R = op.R[0]
    r = R[0, 1]
    quad = 4 * R[0, 0] ** 2 + 4 * R[1, 1] ** 2 + 8 * r ** 2
    bound = 2.0 ** -19 * quad * 3.1  # z: the sums s_it are about 2 R
    for _ in range(10000):
        off = x * rng.uniform(0.5, 1.0)
        E = np.array([[C[0, 0] * r + r, C[0, 1] * r - r + off], [C[1, 0] * r - r - off, C[1, 1] * r + r]])
        E = 1.0 - (1.0 - E)
        s = lambda i, j: Fraction(E[i, j]) + Fraction(E[j, i]) - 2 * int(C[i, j]) * Fraction(r)  # noqa: E731
        # D = -2 r (s_00 + s_11 - 2 s_01) + quad = 1.6 bounds
        E[0, 0] = (float(2 * s(0, 1) - s(1, 1)) + (quad - 1.6 * bound) / (2 * r)) / 2 + C[0, 0] * r
        E = 1.0 - (1.0 - E)
        d = lambda i, j: fma(-float(C[i, j]), r, E[i, j])  # noqa: E731
        G = lambda i, t: r * (d(i, t) + d(t, i))  # noqa: E731
        D = 0.0
        for t, u in ((0, 1.0), (1, -1.0)):
            D = fma(u, fma(u, 4.0 * (r * r), -2.0 * (G(0, t) - G(1, t))), D)
        D = fma(4.0, 2.0 * (r * r), D)
        once = lambda i, j: fma(-float(C[i, j]), 2 * r, E[i, j] + E[j, i])  # noqa: E731
        if D < 0.0 and -2.0 * r * (once(0, 0) + once(1, 1) - 2.0 * once(0, 1)) + quad > 1.4 * bound:
            return 1.0 - E
    raise AssertionError("no such target")


@pytest.mark.parametrize("cell,x", [(10, 9e5), (20, 1e2), (50, 1e2), (50, 9e5)])
def test_asymmetric_targets(cell, x):
    """Targets far apart across the diagonal, from a state that meets their mean: the bound does not cover
    the rounding of d_01 + d_10 where they are too far apart, and every proposal is then exact."""
    species = [2 * cell ** 3] * 2
    nbor, sizes = L.neighbors(L.FCC, cell, L.SHELLS_REFERENCE)
    row = int(sizes[0])
    oracle = lambda target: ho.Problem(nbor[:, :row], sizes[:1], species, [1.0], target.reshape(1, 4))  # noqa: E731
    op = oracle(np.zeros((2, 2)))
    occ = op.generate(5, 0, 0)
    C = op.recount(occ)[0]
    if x < 1e3 or cell == 10:  # covered
        r = op.R[0, 0, 1]
        target = 1.0 - (C * r + np.array([[r, x - r], [-x - r, r]]))
    else:
        target = asymmetric_target(op, C, np.random.default_rng(cell), x)
    op = oracle(target)
    want = op.mc(9, 2 << 16, occ, 300, 2, max_rounds=4, trace_cap=4)
    gp = hb.Problem(nbor, sizes, species, [1.0], target.reshape(1, 4))
    for p in (gp, hb.Problem(nbor, sizes, species, [1.0], target.reshape(1, 4), recognize=False)):
        got = hb.local_search(p, 9, 2, occ[None], 300, 2, max_rounds=4, trace_cap=4)
        assert [t[:4] for t in got["trace"][0]] == [t[:4] for t in want["trace"]]
        np.testing.assert_array_equal(got["occ"][0], want["occ"])
        assert got["f2"][0] == want["f2"]
