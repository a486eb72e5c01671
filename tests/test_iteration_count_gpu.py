"""Stats.iterations counts frontiers processed one after the other, as the reference's
`iteration` global does, also where CTAs follow small frontiers through several rounds
between two team barriers: n on a path of n vertices, the number of levels of a breadth-
first run (every frontier is one level), from nps_sssp, the state form, a batch, the
no-allocation form and nps_bfs."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _path(nps, n):
    return nps.convertCSR(n, np.arange(n - 1), np.arange(1, n), np.full(n - 1, 3, np.uint32))


def _dev(cuda_device, g):
    import torch
    return [torch.from_numpy(a.view(np.int32)).to(cuda_device) for a in (g.row_ptr, g.col, g.w)]


def _noalloc(nps, d, g, out, params):
    from importlib import import_module
    st = import_module("nested-parallelism_b200._native").nps_stats()
    p = params.to_c(device_ptrs=True)
    assert nps.lib.nps_sssp_noalloc(*[x.data_ptr() for x in d], g.n, g.m, 0, out.data_ptr(), C.byref(p), C.byref(st)) == 0
    return st.iterations


@pytest.mark.parametrize("n", [2, 32, 33, 34, 65, 1000])
def test_paths_count_their_vertices(nps, cuda_device, n):
    import torch
    g = _path(nps, n)
    d, out = _dev(cuda_device, g), torch.empty(n, dtype=torch.int32, device=cuda_device)
    torch.cuda.synchronize()
    for level in (0, 1, 2, 3):
        for kw in ({}, {"block_size": 128, "ctas_per_sm": 1}, {"local_rounds": 0, "light_heavy": False}):
            p = nps.Params(level=level, **kw)
            assert nps.sssp(g, 0, p)[1].iterations == n
            assert _noalloc(nps, d, g, out, p) == n
            cost = torch.full((n,), nps.INF, dtype=torch.int32, device=cuda_device)
            upd = torch.zeros(n, dtype=torch.uint8, device=cuda_device)
            cost[0], upd[0] = 0, 1
            torch.cuda.synchronize()
            assert nps.sssp_np_consolidate_gpu(*d, cost, upd, n, g.m, params=p).iterations == n
    stats, _ = nps.sssp_batch([nps.Instance(*d, out, n, g.m, 0)], nps.Params(level=2))
    assert stats[0].iterations == n
    assert nps.bfs(g, 0)[1].iterations == n


def test_trees_count_their_levels(nps, oracle, cuda_device):
    """700 chains of one length behind two levels of small rows: the frontier stays as wide
    as they are many, and every CTA that holds some follows them through many rounds."""
    width, length = 700, 75
    twigs = 1 + np.arange(20)
    v = 21 + np.arange(width * length).reshape(length, width)
    s = np.concatenate([np.zeros(20, np.int64), np.repeat(twigs, 35), v[:-1].ravel()])
    d = np.concatenate([twigs, v[0], v[1:].ravel()])
    g = nps.convertCSR(21 + width * length, s, d, np.ones(s.shape[0], np.uint32))
    levels = int(oracle.bfs_levels(g.row_ptr, g.col, 0).max()) + 1
    for level in (0, 1, 2, 3):
        p = nps.bfs_params(level=level, threshold=64)
        assert nps.bfs(g, 0, p)[1].iterations == levels
        assert nps.sssp(g, 0, p)[1].iterations == levels
