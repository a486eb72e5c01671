"""nps_bc on graphs whose levels reach the reference's mark of unvisited vertices (9999):
paths around that length, in one and in both directions, below and above the vertex count
up to which a source fits shared memory, from one source and from several (some of them
shallow).  Bit for bit as the oracle's restatement of bc_cpu.  A vertex on level 9999 that
is taken more often than there is room for ends the call with an error."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _path(nps, n, both):
    a, b = np.arange(n - 1), np.arange(1, n)
    s, d = (np.concatenate([a, b]), np.concatenate([b, a])) if both else (a, b)
    return nps.convertCSR(n, s, d, np.ones(s.shape[0], np.uint32))


@pytest.mark.parametrize("n", [9998, 9999, 10000, 10001, 10002, 12000, 17600, 18500])
@pytest.mark.parametrize("both", [False, True])
def test_paths(nps, oracle, cuda_device, n, both):
    g = _path(nps, n, both)
    for src in ([0], [n // 2, n - 1, 0, 7] + list(range(20, 400, 2))):
        got, st = nps.bc(g, np.array(src))
        want = np.asarray(oracle.bc(g.row_ptr, g.col, src), np.float32)
        assert st.status == 0 and np.array_equal(np.asarray(got, np.float32).view(np.uint32), want.view(np.uint32))


@pytest.mark.parametrize("n,k", [(10100, 5000), (20000, 15000)])
def test_repeated_visits_end_with_an_error(nps, oracle, cuda_device, n, k):
    """k edges from level 9998 to one vertex, where n + 4,096 - 9,999 visits have room; the
    library works on afterwards."""
    s = np.concatenate([np.arange(9998), np.full(k, 9998)])
    d = np.concatenate([np.arange(1, 9999), np.full(k, 9999)])
    g = nps.convertCSR(n, s, d, np.ones(s.shape[0], np.uint32))
    with pytest.raises(nps.NpsError) as ei:
        nps.bc(g, np.array([0]))
    assert ei.value.status == 3
    got, st = nps.bc(g, np.array([1]))  # one level less: every edge counts
    want = np.asarray(oracle.bc(g.row_ptr, g.col, [1]), np.float32)
    assert st.status == 0 and np.array_equal(np.asarray(got, np.float32).view(np.uint32), want.view(np.uint32))
