"""Populations ahead leave other requests room: a request that does not fit the
server's arena or its level's ring with several is admitted with one."""
import numpy as np
import pytest

import pyhea_b200 as hb
from pyhea_b200 import lattice as L
from pyhea_b200 import workloads as W

pytestmark = pytest.mark.gpu

P, TASKS, DEPTH = 4, 64, 4
SPECIES = W.dirichlet_counts(np.random.default_rng(3), 4, L.num_sites(L.BCC, 12))
TARGET = W.projected_target(np.random.default_rng(4), SPECIES / SPECIES.sum(), 0.1)


def submit(srv, seed, iters, tolerance=-1.0):
    return srv.submit_lattice(L.BCC, 12, SPECIES, W.WEIGHTS, TARGET,
                              dict(num_solutions=P, total_iter=iters, parallel_task=TASKS, converge_depth=DEPTH,
                                   seed=seed), tolerance=tolerance)


def one_population_bytes():
    srv = hb.Server(arena_bytes=64 << 20)
    rid = submit(srv, 1, 1)
    srv.drain()
    size = srv.result(rid)[2]["device_bytes"]
    srv.close()
    return size


def serve(srv, count):
    """Submits `count` requests of six iterations; how many the first step admits, and their results."""
    ids = [submit(srv, 100 + i, 6) for i in range(count)]
    srv.step()
    admitted = count - srv.status()["queued"]
    srv.drain()
    got = [srv.result(i) for i in ids]
    srv.close()
    return admitted, got


def check(got):
    pb = hb.Problem.from_lattice(L.BCC, 12, SPECIES, W.WEIGHTS, TARGET)
    for i, r in enumerate(got):
        occ, fit, _ = hb.search(pb, P, 6, TASKS, DEPTH, seed=100 + i)
        np.testing.assert_array_equal(r[0], occ)
        np.testing.assert_array_equal(r[1], fit)


@pytest.mark.parametrize("count,room", [(2, 3.6), (3, 4.7), (3, 5.7), (2, 6.5)])
def test_arena_room(count, room):
    """With W populations ahead a request takes about (W + 1) / 2 of its room with one: four of them and
    then one each, where the next would have waited for the first."""
    admitted, got = serve(hb.Server(arena_bytes=int(room * one_population_bytes()), slice_ms=0.05), count)
    assert admitted == count
    check(got)


@pytest.mark.parametrize("count,ring_jobs", [(6, 128), (10, 128), (2, 16)])
def test_ring_room(count, ring_jobs):
    """A request holds 2 W P of ring_jobs at its level: two of four populations fill half of 128."""
    admitted, got = serve(hb.Server(arena_bytes=256 << 20, ring_jobs=ring_jobs, slice_ms=0.05), count)
    assert admitted == count
    check(got)


def test_a_lone_request_takes_populations_ahead():
    srv = hb.Server(arena_bytes=256 << 20)
    rid = submit(srv, 7, 6)
    srv.drain()
    assert srv.result(rid)[2]["device_bytes"] > 2 * one_population_bytes()
    srv.close()
