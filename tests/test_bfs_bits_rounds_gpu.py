"""nps_bfs with its levels in step (from 16 M edges at the grid level, 4 M at the block and
hybrid levels), and where they hand over to CTA rounds: paths that leave a uniform graph
after its last large level, so that one, two or every CTA of the team holds part of the
first small frontier, at every CTA size and level, and back again to a second large
frontier behind the paths; a power-law graph from a hub and a leaf; vertex counts around a
word of bits; a head outside the graph.  Exact against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def core(nps):
    return nps.gen_uniform(300_000, 16_200_000, 10, 8)


@pytest.mark.parametrize("paths,length", [(1, 90), (2, 7), (900, 33), (20000, 5)])
def test_handover_to_rounds_and_back(nps, oracle, cuda_device, core, paths, length):
    """`paths` paths of `length` vertices from the core's first vertices; the last vertex of
    the first one has 30,000 heads, so the frontier is large again."""
    n, fan = core.n + paths * length, 30000
    grid = core.n + np.arange(paths * length).reshape(length, paths)
    chain = np.concatenate([np.arange(paths)[None, :], grid])
    s = np.concatenate([np.repeat(np.arange(core.n), core.degrees()), chain[:-1].ravel(), np.full(fan, chain[-1, 0])])
    d = np.concatenate([core.col, chain[1:].ravel(), n + np.arange(fan)])
    g = nps.convertCSR(n + fan, s, d, np.ones(s.shape[0], np.uint32))
    src = core.n - 1
    want = oracle.bfs_levels(g.row_ptr, g.col, src)
    for level, bs in ((0, 512), (1, 128), (2, 128), (2, 256), (2, 512), (3, 512)):
        for ctas in (0, 1):
            got, st = nps.bfs(g, src, nps.bfs_params(level=level, block_size=bs, ctas_per_sm=ctas, block_threshold=128,
                                                     grid_threshold=1024))
            assert st.status == 0 and np.array_equal(got, want)


def test_power_law(nps, oracle, cuda_device):
    g = nps.gen_rmat(20, 17, seed=4)
    assert g.m >= 16_000_000
    leaf = int(np.flatnonzero((g.degrees() > 0) & (g.degrees() < 3))[5])
    for src in (g.source, leaf):
        want = oracle.bfs_levels(g.row_ptr, g.col, src)
        for level, bs, sort in ((2, 128, 0), (2, 512, 0), (2, 512, 1), (2, 512, -1), (1, 256, 0), (3, 256, 0)):
            got, st = nps.bfs(g, src, nps.bfs_params(level=level, block_size=bs, sort_at_push=sort))
            assert st.status == 0 and np.array_equal(got, want)
            assert st.reached == int((want < nps.BFS_UNDEFINED).sum())


@pytest.mark.parametrize("n", [999_999, 1_000_001, 1_000_031, 1_000_032])
def test_vertex_counts(nps, oracle, cuda_device, n):
    g = nps.gen_uniform(n, 16_100_000, 10, n)
    for src in (0, n - 1):
        assert np.array_equal(nps.bfs(g, src)[0], oracle.bfs_levels(g.row_ptr, g.col, src))


def test_a_head_outside_the_graph_is_reported(nps, cuda_device, core):
    import torch
    col = core.col.copy()
    col[core.row_ptr[0]] = core.n
    t = [torch.from_numpy(a.view(np.int32)).to(cuda_device) for a in (core.row_ptr, col)]
    out = torch.empty(core.n, dtype=torch.int32, device=cuda_device)
    torch.cuda.synchronize()
    with pytest.raises(nps.NpsError) as ei:
        nps.bfs_device(*t, core.n, core.m, 0, out)
    assert ei.value.status == 7
