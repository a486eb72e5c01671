"""Host-pointer calls in a process of one host thread, which copy pageable arrays plainly
instead of through slots that the threads fill.  Exact against the oracle."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

CODE = """
import importlib, sys
sys.path[:0] = ["{root}", "{root}/oracle"]
import numpy as np, oracle
nps = importlib.import_module("nested-parallelism_b200")
g = nps.gen_rmat(18, 4, seed=2)
for k in range(2):
    got, st = nps.sssp(g, g.source, nps.Params(level=2))
    assert st.status == 0 and np.array_equal(got, oracle.sssp_heap(g.row_ptr, g.col, g.w, g.source))
    assert np.array_equal(nps.bfs(g)[0], oracle.bfs_levels(g.row_ptr, g.col, g.source))
print("same")
"""


@pytest.mark.parametrize("threads", ["1", "2"])
def test_few_host_threads(cuda_device, threads):
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", CODE.format(root=root)], capture_output=True, text=True, timeout=300,
                       env=dict(os.environ, OMP_NUM_THREADS=threads))
    assert r.returncode == 0 and r.stdout.strip() == "same", r.stderr
