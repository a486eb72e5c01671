"""nps_bfs where the levels in step (graphs of at least 4 M edges) hand over to CTA rounds:
paths that leave a uniform graph after its last large level, so that one, two or every
CTA of the team holds part of the first small frontier, at every CTA size and level, and
back again to a second large frontier behind the paths.  Exact against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def core(nps):
    return nps.gen_uniform(300_000, 4_200_000, 10, 8)


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
