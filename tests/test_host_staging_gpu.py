"""Host-pointer calls whose arrays cross through the pinned slots (pageable arrays of at
least 1 MiB, slots of 2 MiB, four of them): sizes around one slot, one round of slots and
the limit, pageable and pinned arrays, narrow and wide weights, for nps_sssp and nps_bfs,
twice on the same context with other contents.  Exact against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MIB = (1 << 20) // 4  # int32 entries per MiB


@pytest.mark.parametrize("n", [MIB - 2, MIB - 1, MIB, MIB + 1, 2 * MIB, 2 * MIB + 3, 8 * MIB - 1, 8 * MIB + 5])
def test_sizes_around_the_slots(nps, oracle, cuda_device, n):
    """n distances out, n + 1 offsets and about n edges in."""
    rng = np.random.default_rng(n)
    for wmax in (200, 1 << 20):
        dst = np.concatenate([np.arange(1, n), rng.integers(0, n, 1000)])
        src = np.concatenate([rng.integers(0, np.arange(1, n)), rng.integers(0, n, 1000)])
        g = nps.convertCSR(n, src, dst, rng.integers(1, wmax, dst.shape[0]).astype(np.uint32))
        want = oracle.sssp_heap(g.row_ptr, g.col, g.w, 0)
        got, st = nps.sssp(g, 0, nps.Params(level=2))
        assert st.status == 0 and np.array_equal(got, want)
    lv, _ = nps.bfs(g, 0)
    assert np.array_equal(lv, oracle.bfs_levels(g.row_ptr, g.col, 0))


def test_pinned_arrays(nps, oracle, cuda_device):
    import torch
    g = nps.gen_rmat(18, 8, seed=2)
    want = oracle.sssp_heap(g.row_ptr, g.col, g.w, g.source)
    pin = [torch.from_numpy(a.view(np.int32).copy()).pin_memory() for a in (g.row_ptr, g.col, g.w)]
    h = nps.Graph(pin[0].numpy(), pin[1].numpy(), pin[2].numpy().view(np.uint32), g.source)
    out = torch.empty(g.n, dtype=torch.int32).pin_memory().numpy().view(np.uint32)
    for graph, o in ((h, out), (g, out), (h, None), (g, None)):
        got, _ = nps.sssp(graph, params=nps.Params(level=2), out=o)
        assert np.array_equal(got, want)
