"""CTA rounds of the persistent kernel (iterations with few frontier vertices per CTA)
at the sizes where they can go wrong: paths around the round limit and around its
multiples, stars around the stop and capacity of a CTA's queue, rows around the length
that leaves for the grid-tier list, frontiers around the seed limit, at every level,
with and without the light/heavy split, from a source and from a state, alone and in a
batch.  Distances equal the oracle's heap Dijkstra exactly."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _path(nps, n):
    return nps.convertCSR(n, np.arange(n - 1), np.arange(1, n), np.arange(1, n).astype(np.uint32) % 7 + 1)


def _stars(nps, leaves, hubs=3):
    """A chain of hubs, each with `leaves` leaves that lead to the next hub: every hub's
    leaves join one round's queue, and every leaf lowers the next hub again."""
    n = hubs * (leaves + 1) + 1
    s, d, w = [], [], []
    for h in range(hubs):
        base = h * (leaves + 1)
        leaf = base + 1 + np.arange(leaves)
        s += [np.full(leaves, base), leaf]
        d += [leaf, np.full(leaves, base + leaves + 1)]
        w += [1 + np.arange(leaves), 3 * leaves - 2 * np.arange(leaves)]
    return nps.convertCSR(n, np.concatenate(s), np.concatenate(d), np.concatenate(w).astype(np.uint32))


def _check(nps, oracle, g, p, src=0):
    want = oracle.sssp_heap(g.row_ptr, g.col, g.w, src)
    for _ in range(3):
        got, st = nps.sssp(g, src, p)
        assert st.status == 0 and np.array_equal(got, want)
        assert st.reached == int((want < nps.INF).sum())


@pytest.mark.parametrize("n", [2, 31, 32, 33, 34, 64, 65, 1000])
@pytest.mark.parametrize("delta,split", [(0, False), (4, True), (16, False)])
def test_paths_around_the_round_limit(nps, oracle, cuda_device, n, delta, split):
    for bs in (128, 512):
        _check(nps, oracle, _path(nps, n), nps.Params(level=2, block_size=bs, delta=delta, light_heavy=split))


@pytest.mark.parametrize("leaves", [1, 64, 127, 128, 129, 255, 256, 257, 600])
@pytest.mark.parametrize("level", [0, 1, 2, 3])
def test_stars_around_the_queue_and_row_limits(nps, oracle, cuda_device, leaves, level):
    g = _stars(nps, leaves)
    for delta, split, bs in ((0, False, 256), (32, True, 256), (100000, True, 128), (0, False, 512)):
        _check(nps, oracle, g, nps.Params(level=level, threshold=32, block_threshold=128, grid_threshold=512,
                                          block_size=bs, delta=delta, light_heavy=split))


@pytest.mark.parametrize("side", [3, 40, 97, 300])
@pytest.mark.parametrize("delta,split", [(0, False), (256, True), (4096, True), (4096, False)])
def test_grids(nps, oracle, cuda_device, side, delta, split):
    g = nps.gen_grid(side, side + 1, 0.05, 1000, side)
    for level, bs, ctas in ((2, 256, 0), (1, 512, 0), (0, 128, 1)):
        _check(nps, oracle, g, nps.Params(level=level, block_size=bs, ctas_per_sm=ctas, delta=delta,
                                          light_heavy=split))


def test_weights_near_the_limit(nps, oracle, cuda_device):
    """Tentative distances that reach 2^30 leave their heads unreached."""
    w = np.array([2**29, 2**29 - 1, 2, 2**30 - 1, 5], np.uint32)
    g = nps.convertCSR(6, [0, 1, 2, 0, 4], [1, 2, 3, 4, 5], w)
    for delta in (0, 1 << 20):
        _check(nps, oracle, g, nps.Params(level=2, delta=delta))


@pytest.mark.parametrize("count", [1, 4735, 4736, 4737, 20000])
def test_state_frontiers_around_the_seed_limit(nps, oracle, cuda_device, count):
    """`count` vertices flagged in the initial state (the limit is 32 per CTA: 4736 with one CTA per SM)."""
    import torch
    g = nps.gen_uniform(30011, 120044, 50, 9)
    rng = np.random.default_rng(count)
    cost = np.full(g.n, nps.INF, np.uint32)
    flag = np.zeros(g.n, np.uint8)
    at = rng.choice(g.n, count, replace=False)
    cost[at] = rng.integers(0, 40, count)
    flag[at] = 1
    want = oracle.sssp_state(g.row_ptr, g.col, g.w, cost.copy(), flag.copy())
    want = want[0] if isinstance(want, tuple) else want
    t = [torch.from_numpy(a.view(np.int32)).to(cuda_device) for a in (g.row_ptr, g.col, g.w, cost)]
    upd = torch.from_numpy(flag).to(cuda_device)
    torch.cuda.synchronize()
    for delta in (0, 16):
        c, u = t[3].clone(), upd.clone()
        torch.cuda.synchronize()
        st = nps.sssp_np_consolidate_gpu(t[0], t[1], t[2], c, u, g.n, g.m,
                                         params=nps.Params(level=2, ctas_per_sm=1, delta=delta))
        assert st.status == 0 and int(u.sum()) == 0
        assert np.array_equal(c.cpu().numpy().view(np.uint32), want)


def test_batch_of_small_graphs(nps, oracle, cuda_device):
    import torch
    gs = [_path(nps, 500), _stars(nps, 130), nps.gen_grid(60, 50, 0.05, 100, 4), nps.gen_rmat(12, 8, seed=6)]
    dev = []
    for g in gs:
        t = [torch.from_numpy(a.view(np.int32)).to(cuda_device) for a in (g.row_ptr, g.col, g.w)]
        dev.append((*t, torch.empty(g.n, dtype=torch.int32, device=cuda_device)))
    torch.cuda.synchronize()
    for delta, split in ((0, False), (64, True)):
        for ctas in (0, 1):
            stats, _ = nps.sssp_batch([nps.Instance(*d, g.n, g.m, 0) for d, g in zip(dev, gs)],
                                      nps.Params(level=2, delta=delta, light_heavy=split, ctas_per_sm=ctas))
            for d, g, st in zip(dev, gs, stats):
                assert st.status == 0
                assert np.array_equal(d[3].cpu().numpy().view(np.uint32),
                                      oracle.sssp_heap(g.row_ptr, g.col, g.w, 0))


def test_malformed_rows_and_heads_are_reported(nps, cuda_device):
    """A head outside the graph, and row bounds that decrease, met in a round."""
    import torch
    g = _path(nps, 40)
    for what in ("head", "row"):
        row, col = g.row_ptr.copy(), g.col.copy()
        if what == "head":
            col[20] = 40
        else:
            row[21] = 5
        t = [torch.from_numpy(a.view(np.int32)).to(cuda_device) for a in (row, col, g.w)]
        out = torch.empty(g.n, dtype=torch.int32, device=cuda_device)
        torch.cuda.synchronize()
        with pytest.raises(nps.NpsError) as ei:
            nps.sssp_device(*t, g.n, g.m, 0, out, nps.Params(level=2))
        assert ei.value.status == 7


@pytest.mark.parametrize("ef", [2, 8, 24])
@pytest.mark.parametrize("level", [0, 1, 2])
def test_rounds_pause_where_rows_are_listed(nps, oracle, cuda_device, ef, level):
    """Long rows met in rounds (power-law graphs, from a hub and from a leaf) and a road
    with hubs, so that rounds run, pause and run again; average degrees from 2 to 24 move
    the seed limit."""
    g = nps.gen_rmat(12, ef, seed=ef)
    leaf = int(np.flatnonzero((g.degrees() > 0) & (g.degrees() < 4))[0])
    n = 4000
    hubs = np.arange(0, n, 500)
    s = np.concatenate([np.arange(n - 1), np.repeat(hubs, 200)])
    d = np.concatenate([np.arange(1, n), (np.repeat(hubs, 200) + np.tile(np.arange(200), hubs.size) * 7 + 2) % n])
    road = nps.convertCSR(n, s, d, (np.arange(s.size) % 90 + 1).astype(np.uint32))
    for delta in (0, 64):
        p = nps.Params(level=level, threshold=32, delta=delta)
        _check(nps, oracle, g, p, g.source)
        _check(nps, oracle, g, p, leaf)
        _check(nps, oracle, road, p)
