"""nps_bfs with its levels in step (graphs of at least 4 M edges, unordered): power-law and
uniform graphs from a hub, a leaf and a vertex behind a long path, vertex counts around a
word of bits, every level, grid-tier rows sorted at push or not, and a head outside the
graph.  Exact against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _tail(nps, g, length):
    """g, a path that leads into its hub and a path that leaves one of the hub's heads."""
    n = g.n + 2 * length
    src = np.repeat(np.arange(g.n), g.degrees())
    a, b = g.n + np.arange(length), g.n + length + np.arange(length)
    head = g.col[g.row_ptr[g.source]]
    s = np.concatenate([src, a, [head], b[:-1]])
    d = np.concatenate([g.col, a[1:], [g.source], [b[0]], b[1:]])
    return nps.convertCSR(n, s, d, np.ones(s.shape[0], np.uint32)), int(a[0])


@pytest.fixture(scope="module")
def rmat(nps):
    return nps.gen_rmat(18, 20, seed=4)


@pytest.mark.parametrize("level", [0, 1, 2, 3])
@pytest.mark.parametrize("sort", [0, 1, -1])
def test_power_law(nps, oracle, cuda_device, rmat, level, sort):
    assert rmat.m >= 4_000_000
    leaf = int(np.flatnonzero((rmat.degrees() > 0) & (rmat.degrees() < 3))[5])
    for src in (rmat.source, leaf):
        want = oracle.bfs_levels(rmat.row_ptr, rmat.col, src)
        for bs in (128, 512):
            for _ in range(2):
                got, st = nps.bfs(rmat, src, nps.bfs_params(level=level, block_size=bs, sort_at_push=sort, threshold=32,
                                                            block_threshold=128, grid_threshold=1024))
                assert st.status == 0 and np.array_equal(got, want)
                assert st.reached == int((want < nps.BFS_UNDEFINED).sum())


@pytest.mark.parametrize("length", [3, 4, 5, 40, 333])
def test_long_paths_around_a_power_law_graph(nps, oracle, cuda_device, rmat, length):
    g, start = _tail(nps, rmat, length)
    for src in (start, rmat.source):
        want = oracle.bfs_levels(g.row_ptr, g.col, src)
        for _ in range(2):
            assert np.array_equal(nps.bfs(g, src)[0], want)


@pytest.mark.parametrize("n", [999_999, 1_000_000, 1_000_001, 1_000_031, 1_000_032])
def test_vertex_counts(nps, oracle, cuda_device, n):
    g = nps.gen_uniform(n, 4_100_000, 10, n)
    for src in (0, n - 1):
        assert np.array_equal(nps.bfs(g, src)[0], oracle.bfs_levels(g.row_ptr, g.col, src))


def test_a_head_outside_the_graph_is_reported(nps, cuda_device, rmat):
    import torch
    col = rmat.col.copy()
    col[rmat.row_ptr[rmat.source]] = rmat.n
    t = [torch.from_numpy(a.view(np.int32)).to(cuda_device) for a in (rmat.row_ptr, col)]
    out = torch.empty(rmat.n, dtype=torch.int32, device=cuda_device)
    torch.cuda.synchronize()
    with pytest.raises(nps.NpsError) as ei:
        nps.bfs_device(*t, rmat.n, rmat.m, rmat.source, out)
    assert ei.value.status == 7
