"""nps_bc's shared-memory kernel at the sizes where it can go wrong: graphs around the
vertex counts where the CTA size changes and where a graph no longer fits shared memory,
rows around the long-row limit (32) and whole batches of heads (32, 64, 95), sums that
cross binades or meet ties, path counts that wrap to negative and to zero, and more than
256 levels.  Bit for bit as the oracle's restatement of bc_cpu, NaNs as NaNs."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _same(a, b):
    a, b = np.asarray(a, np.float32), np.asarray(b, np.float32)
    bits = a.view(np.uint32) == b.view(np.uint32)
    return bool(np.all(bits | (np.isnan(a) & np.isnan(b))))


def _graph(nps, n, s, d):
    s, d = np.concatenate(s).astype(np.int64), np.concatenate(d).astype(np.int64)
    return nps.convertCSR(n, s, d, np.ones(s.shape[0], np.uint32))


@pytest.mark.parametrize("n", [1, 2, 31, 33, 2100, 2200, 8600, 8900, 9000, 16384, 17000, 17100, 17700, 18200, 20000])
def test_vertex_counts(nps, oracle, cuda_device, n):
    g = nps.gen_uniform(n, 5 * n, 10, n) if n > 1 else nps.convertCSR(1, [], [], [])
    src = np.unique(np.linspace(0, n - 1, 12).astype(np.int64))
    b, st = nps.bc(g, src)
    assert st.status == 0 and _same(b, oracle.bc(g.row_ptr, g.col, src))


@pytest.mark.parametrize("k", [1, 31, 32, 33, 63, 64, 65, 95, 96, 97, 127, 128, 129, 1000])
def test_row_lengths(nps, oracle, cuda_device, k):
    """A source, two hubs with k heads each (every third one off the next level), heads
    with 0 to 6 heads of their own, so the terms are fractions of many sizes."""
    rng = np.random.default_rng(k)
    hub, heads = np.array([1, 2]), 3 + np.arange(k)
    tails = 3 + k + np.arange(7 * k)
    s = [np.zeros(2), np.repeat(hub, k), np.zeros((k + 2) // 3)]
    d = [hub, np.tile(heads, 2), heads[::3]]  # heads[::3] are on the hubs' own level
    cnt = rng.integers(0, 7, k)
    s.append(np.repeat(heads, cnt))
    d.append(rng.choice(tails, int(cnt.sum())))
    g = _graph(nps, 3 + 8 * k, s, d)
    src = np.array([0, 1, 2, 0])
    assert _same(nps.bc(g, src)[0], oracle.bc(g.row_ptr, g.col, src))


@pytest.mark.parametrize("width,layers", [(40, 4), (40, 9), (64, 7), (33, 14), (7, 300)])
def test_layers_and_wrapping_path_counts(nps, oracle, cuda_device, width, layers):
    """Complete bipartite layers: width^L paths, which wrap (64^6 = 2^36 is zero in an int)."""
    n = 1 + width * layers
    base = 1 + width * np.arange(layers - 1)
    a, b = np.meshgrid(np.arange(width), np.arange(width), indexing="ij")
    s = [np.zeros(width)] + [x + a.ravel() for x in base]
    d = [1 + np.arange(width)] + [x + width + b.ravel() for x in base]
    g = _graph(nps, n, s, d)
    src = np.array([0, 1, n - 1])
    assert _same(nps.bc(g, src)[0], oracle.bc(g.row_ptr, g.col, src))


@pytest.mark.parametrize("heads", [40, 300, 5000])
def test_ties_and_binades(nps, oracle, cuda_device, heads):
    """A hub whose heads end it in dyadic terms: sums cross binades at every doubling, and a
    chain behind some heads makes terms of 2^k + 1, ties where the sum is large."""
    s, d, nxt = [np.zeros(1), np.full(heads, 1)], [np.ones(1), 2 + np.arange(heads)], 2 + heads
    for i, ln in ((0, 1), (7, 3), (heads // 2, 64), (heads - 1, 1000), (heads - 2, 8000)):
        c = np.concatenate([[2 + i], nxt + np.arange(ln)])
        s.append(c[:-1])
        d.append(c[1:])
        nxt += ln
    # halves: vertices reached from two heads
    for i in range(0, heads - 9, 5):
        s.append(np.array([2 + i, 3 + i]))
        d.append(np.array([nxt, nxt]))
        nxt += 1
    g = _graph(nps, nxt, s, d)
    src = np.array([0, 1])
    assert _same(nps.bc(g, src)[0], oracle.bc(g.row_ptr, g.col, src))


def test_every_source_of_a_power_law_graph(nps, oracle, cuda_device):
    g = nps.gen_rmat(12, 16, seed=21)
    assert _same(nps.bc(g)[0], oracle.bc(g.row_ptr, g.col))
