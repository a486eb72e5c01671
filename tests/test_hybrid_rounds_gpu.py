"""CTA rounds at the hybrid level: rows from 128 edges on join the grid-tier list there too,
also below the grid threshold, so many more of them in one iteration than there are rows
of that threshold.  Distances equal the oracle's heap Dijkstra."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("length", [126, 127, 128, 129, 400])
@pytest.mark.parametrize("threshold", [1, 64, 128, 200])
def test_rows_below_the_grid_threshold(nps, oracle, cuda_device, length, threshold):
    """40 hubs on the ends of paths of different lengths, so that they are met in one round
    or in several, each with `length` edges back into the graph."""
    rng = np.random.default_rng(length)
    hubs, n = 40, 6000
    s, d, at = [], [], 1
    for h in range(hubs):
        ln = 3 if h % 2 else 1 + h
        chain = np.concatenate([[0], at + np.arange(ln)])
        s += [chain[:-1], np.full(length, chain[-1])]
        d += [chain[1:], rng.integers(1, n, length)]
        at += ln
    s, d = np.concatenate(s), np.concatenate(d)
    g = nps.convertCSR(n, s, d, (1 + np.arange(s.size) % 9).astype(np.uint32))
    want = oracle.sssp_heap(g.row_ptr, g.col, g.w, 0)
    for delta, split, bs in ((0, False, 256), (8, True, 256), (8, False, 128), (1000, True, 512)):
        got, st = nps.sssp(g, 0, nps.Params(level=3, threshold=threshold, block_threshold=max(256, threshold),
                                            grid_threshold=4096, block_size=bs, delta=delta, light_heavy=split))
        assert st.status == 0 and np.array_equal(got, want)
