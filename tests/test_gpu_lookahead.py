"""Populations searched ahead of the survivors: whole searches whose iterations
outnumber the populations in flight (their slots are reused), plans run again
and from several threads, and calls after the cached streams were given back,
all equal to the oracle bit for bit."""
import threading

import numpy as np
import pytest

import pyhea_b200 as hb
from oracle import hea_oracle as ho
from pyhea_b200 import lattice as L
from pyhea_b200 import workloads as W

pytestmark = pytest.mark.gpu


def case(seed, lattice=L.BCC, cell=3, species=(20, 17, 17)):
    st = W.small_case(lattice=lattice, cell=cell, species=species, shells=2, seed=seed)
    nbor, sizes = st.neighbors()
    return (hb.Problem(nbor, sizes, st.species, st.weight, st.target),
            ho.Problem(nbor, sizes, st.species, st.weight, st.target))


def same(got, want):
    occ, fit = got[0], got[1]
    wocc, wf2 = want[0], want[1]
    np.testing.assert_array_equal(occ, wocc)
    np.testing.assert_array_equal(fit, np.sqrt(wf2))


@pytest.mark.parametrize("iters", [1, 2, 16, 17, 35])
def test_iterations_around_the_populations_in_flight(iters):
    gp, op = case(iters)
    same(hb.search(gp, 3, iters, 24, 3, seed=11 + iters), op.hcs(11 + iters, 3, iters, 24, 3))


def test_cluster_path_reuses_population_slots():
    gp, op = case(5)
    same(hb.search(gp, 2, 19, 40, 2, seed=3, hbm_occupancy=True), op.hcs(3, 2, 19, 40, 2))


def test_plan_runs_again():
    gp, op = case(7)
    plan = hb.Plan(gp, 4, 18, 16, 3)
    for seed in (1, 2, 1):
        plan.run(seed)
        same(plan.read(), op.hcs(seed, 4, 18, 16, 3))
    plan.close()


def test_a_tuned_size_is_kept_for_plans_with_as_much_in_flight():
    """The size tuned for one iteration (64 searches at once) is not taken by a plan of sixteen, whose
    default is smaller CTAs, and the other way round; both give the same search."""
    st = W.small_case(lattice=L.BCC, cell=10, species=(700, 650, 650), shells=3, seed=1)
    pb = st.problem()
    default = {}
    for iters in (1, 16):
        with_default = hb.Plan(pb, 64, iters, 512, 2)
        default[iters] = with_default.local_search_block
        with_default.close()
    assert default[1] == 512 and default[16] == 256
    hb.Plan(pb, 64, 1, 512, 2, autotune=True).close()
    plan = hb.Plan(pb, 64, 16, 512, 2)
    assert plan.local_search_block == default[16]
    hb.Plan(pb, 64, 16, 512, 2, autotune=True).close()
    one = hb.Plan(pb, 64, 1, 512, 2, autotune=True)
    again = hb.Plan(pb, 64, 1, 512, 2)
    assert again.local_search_block == one.local_search_block
    for p in (plan, one, again):
        p.close()


@pytest.mark.parametrize("P,iters,tasks", [(5, 1, 300), (5, 0, 300), (40, 18, 512), (75, 9, 600), (3, 2, 130)])
def test_tuned_plans_search_the_same(P, iters, tasks):
    """Other sizes than the default are tried in the plan's own slots, whatever its iterations."""
    gp, op = case(31)
    plan = hb.Plan(gp, P, iters, tasks, 2, autotune=True)
    passes = -(-tasks // 256)
    whole, equal = min(512, -(-tasks // 32) * 32), -(-(-(-tasks // passes)) // 32) * 32  # one pass; equal passes
    assert plan.local_search_block in {whole, equal, 256, 128}
    for seed in (3, 4):
        plan.run(seed)
        same(plan.read(), op.hcs(seed, P, iters, tasks, 2))
    plan.close()


def test_threads_share_the_stream_cache():
    gp, op = case(9)
    want = {s: op.hcs(s, 3, 4, 24, 3) for s in range(6)}
    got, errors = {}, []

    def work(s):
        try:
            for _ in range(4):
                got[s] = hb.search(gp, 3, 4, 24, 3, seed=s)
        except Exception as e:  # reported by the main thread
            errors.append(e)

    threads = [threading.Thread(target=work, args=(s,)) for s in want]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors
    for s in want:
        same(got[s], want[s])


def test_after_release_of_cached_memory():
    gp, op = case(13)
    for _ in range(2):
        same(hb.search(gp, 3, 3, 24, 3, seed=4), op.hcs(4, 3, 3, 24, 3))
        hb.lib.hea_release_cached_memory()


@pytest.mark.parametrize("iters", [0, 1, 3, 4, 5, 11])
def test_batch_populations_ahead(iters):
    """Iterations around the populations a batch keeps in flight; the first structure has two more."""
    cases = [case(20 + i, species=(18, 18, 18)) for i in range(4)]
    its = [iters + 2 if i == 0 else iters for i in range(4)]
    b = hb.Batch([gp for gp, _ in cases],
                 [dict(num_solutions=3 + i, total_iter=its[i], parallel_task=24, converge_depth=3) for i in range(4)])
    for seeds in ((5, 6, 7, 8), (15, 6, 17, 8)):
        b.run(seeds)
        for i, (_, op) in enumerate(cases):
            same(b.read(i), op.hcs(seeds[i], 3 + i, its[i], 24, 3))
    b.close()


@pytest.mark.parametrize("tasks", [16, 32, 37, 64, 100, 256, 300])
def test_batch_counts_each_job_once(tasks):
    """Rounds, evaluations and accepts for task counts that leave warps of a CTA idle or part full."""
    gp, op = case(3, lattice=L.BCC, cell=5, species=(100, 75, 75))
    b = hb.Batch([gp], [dict(num_solutions=7, total_iter=2, parallel_task=tasks, converge_depth=4)])
    b.run([9])
    want = op.hcs(9, 7, 2, tasks, 4)
    same(b.read(0), want)
    assert [int(v) for v in b.tallies()[0]] == [want[2]["rounds"], want[2]["evals"], want[2]["accepts"]]
    b.close()


def test_served_requests_with_populations_ahead():
    cases = [case(40 + i) for i in range(5)]
    srv = hb.Server(slice_ms=0.2)
    prm = [dict(num_solutions=3 + i, total_iter=2 * i + 1, parallel_task=24, converge_depth=3, seed=60 + i)
           for i in range(5)]
    ids = [srv.submit(gp, q) for (gp, _), q in zip(cases, prm)]
    srv.drain()
    for rid, (_, op), q in zip(ids, cases, prm):
        same(srv.result(rid), op.hcs(q["seed"], q["num_solutions"], q["total_iter"], 24, 3))
    srv.close()


@pytest.mark.parametrize("tasks", [16, 64, 300])
def test_batch_counts_each_job_once_in_many_runs(tasks):
    """Several structures with short jobs: CTAs of every structure take and wait for jobs at once, and
    each run's tallies are the oracle's."""
    cases = [case(70 + i, cell=3 + i % 3, species=[(20, 17, 17), (48, 40, 40), (100, 75, 75)][i % 3]) for i in range(6)]
    b = hb.Batch([gp for gp, _ in cases],
                 [dict(num_solutions=40, total_iter=6, parallel_task=tasks, converge_depth=2)] * len(cases))
    want = [op.hcs(9 + i, 40, 6, tasks, 2)[2] for i, (_, op) in enumerate(cases)]
    want = [[w["rounds"], w["evals"], w["accepts"]] for w in want]
    for _ in range(30):
        b.run([9 + i for i in range(len(cases))])
        np.testing.assert_array_equal(b.tallies(), want)
    b.close()
