"""Device memory of the populations searched ahead: what a batch takes where the
device has little, and what many plans take together."""
import gc

import numpy as np
import pytest
import torch

import pyhea_b200 as hb
from pyhea_b200 import lattice as L
from pyhea_b200 import workloads as W

pytestmark = pytest.mark.gpu

MIB = 1 << 20
GIB = 1 << 30


def free_bytes():
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def give_back():
    gc.collect()
    hb.lib.hea_release_cached_memory()
    torch.cuda.empty_cache()


def structure(lattice, cell, types, seed=0):
    rng = np.random.default_rng(seed)
    species = W.dirichlet_counts(rng, types, L.num_sites(lattice, cell))
    target = W.projected_target(rng, species / species.sum(), 0.1)
    return hb.Problem.from_lattice(lattice, cell, species, W.WEIGHTS, target)


def test_a_batch_short_of_memory_takes_what_fits():
    """Four populations ahead do not fit and two do: the batch takes more than the one it needs, and
    searches the same."""
    pb = structure(L.BCC, 30, 4)  # 54 000 sites: 486 KB a slot
    P = 256
    slot = P * 9 * pb.num_sites  # one population's histograms and occupancies
    prm = [dict(num_solutions=P, total_iter=4, parallel_task=64, converge_depth=1, max_rounds=2)]

    def taken():
        give_back()
        before = free_bytes()
        b = hb.Batch([pb], prm)
        used = before - free_bytes()
        b.run([5])
        got = b.read(0)
        b.close()
        return used, got

    full, want = taken()
    assert full > 4.9 * slot  # survivors and four populations
    give_back()
    spare = int(3.6 * slot)
    block = torch.empty(free_bytes() - spare, dtype=torch.uint8, device="cuda")
    short, got = taken()
    del block
    give_back()
    assert 2.9 * slot < short < 3.6 * slot
    np.testing.assert_array_equal(got[0], want[0])
    np.testing.assert_array_equal(got[1], want[1])


@pytest.mark.parametrize("form", ["plan", "batch"])
def test_many_searches_leave_the_device_its_memory(form):
    """Each alone would search several populations ahead; all together take 16 GiB for those beyond the
    first, and what they return comes back when they close."""
    if form == "plan":
        pb = structure(L.FCC, 80, 3)  # 2 048 000 sites
        count, P = 12, 8
        make = lambda: hb.Plan(pb, P, 16, 64, 2, max_rounds=2)
    else:
        pb = structure(L.FCC, 80, 3)
        count, P = 8, 64
        make = lambda: hb.Batch([pb], [dict(num_solutions=P, total_iter=16, parallel_task=64, converge_depth=1)])
    each = 9 * P * pb.num_sites
    for _ in range(2):
        give_back()
        before = free_bytes()
        kept, used = [], []
        for _ in range(count):
            kept.append(make())
            used.append(before - free_bytes())
        extra = used[-1] - count * 2.2 * each  # beside survivors, one population and the reading buffer
        assert extra < 16 * GIB
        assert used[0] > 3 * each  # the first ones search ahead
        for k in kept:
            k.close()
    give_back()
    assert before - free_bytes() < 64 * MIB


def test_buffers_of_the_last_search_stay_cached():
    """Plans of other shapes fill the block cache; a batch made after them finds its buffers there
    when it is made again, and the cache keeps its bound."""
    give_back()
    start = free_bytes()
    large = structure(L.FCC, 60, 3)  # 864 000 sites
    for P in range(64, 73):  # about 1 GiB each, no shape twice
        hb.Plan(large, P, 1, 64, 2, max_rounds=2).close()
    small = structure(L.BCC, 30, 4)
    make = lambda: hb.Batch([small], [dict(num_solutions=256, total_iter=4, parallel_task=64,  # noqa: E731
                                           converge_depth=1, max_rounds=2)])
    make().close()
    kept = free_bytes()
    assert start - kept < 9 * GIB
    b = make()
    assert kept - free_bytes() < 16 * MIB  # of the batch's 620 MB nothing allocated
    b.close()
    assert abs(kept - free_bytes()) < 16 * MIB
    give_back()
    assert start - free_bytes() < 64 * MIB
