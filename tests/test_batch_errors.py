"""A batch whose structures cannot be prepared reports an error: here the device
memory of a neighbour table, which a machine without a GPU cannot give."""
import subprocess
import sys

import pytest

import pyhea_b200 as hb
from conftest import REPO

PROGRAM = """
import sys
sys.path.insert(0, {repo!r})
import pyhea_b200 as hb
from pyhea_b200 import lattice as L
from pyhea_b200 import workloads as W

st = W.small_case(lattice=L.FCC, cell=4, species=(64, 64, 64, 64), shells=3)
nbor, sizes = st.neighbors()
pb = hb.Problem(nbor, sizes, st.species, st.weight, st.target, recognize={recognize})
try:
    hb.Batch([pb] * {count}, [dict(num_solutions=3, total_iter=2, parallel_task=16, converge_depth=2)] * {count})
except Exception as e:
    print("raised", type(e).__name__, e)
"""


@pytest.mark.skipif(hb.cuda_available(), reason="needs a machine without a GPU")
@pytest.mark.parametrize("recognize", [True, False])
@pytest.mark.parametrize("count", [1, 40])
def test_table_memory_failure_is_an_error(recognize, count):
    """In a process of its own, since the failure once ended it."""
    run = subprocess.run([sys.executable, "-c", PROGRAM.format(repo=REPO, recognize=recognize, count=count)],
                         capture_output=True, text=True, timeout=300)
    assert run.returncode == 0, run.stderr[-500:]
    assert "raised" in run.stdout and "structure 0" in run.stdout, run.stdout
