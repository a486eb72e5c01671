"""nps_color at the sizes where its units can go wrong: rows around the length that makes
a row a unit of its own (64 edges) and around whole chunks (1,024 edges), runs around 32
vertices, and more neighbours without a color than a run's list (384) or a chunk's (1,024)
holds.  Colors equal the oracle's closed form exactly."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _exact(nps, oracle, g, **kw):
    want, it = oracle.color(g.row_ptr, g.col)
    for ctas in (0, 1, 8):
        got, st = nps.color(g, nps.Params(ctas_per_sm=ctas, **kw))
        assert np.array_equal(got, want) and st.iterations == it and st.status == 0
        src = np.repeat(np.arange(g.n), np.diff(g.row_ptr))
        assert st.edges_scanned == int((g.col < src).sum()) and st.buckets == it


@pytest.mark.parametrize("n", [1, 31, 32, 33, 63, 64, 65, 97, 1025, 2050])
def test_complete_order(nps, oracle, cuda_device, n):
    """Every vertex waits for every smaller one: n colors, rows of 0 .. n - 1 edges."""
    s = np.repeat(np.arange(n), np.arange(n))
    d = np.concatenate([np.arange(v) for v in range(n)]) if n > 1 else np.zeros(0, np.int64)
    _exact(nps, oracle, nps.convertCSR(n, s, d.astype(np.int64), np.ones(s.shape[0], np.uint32)))


@pytest.mark.parametrize("length", [62, 63, 64, 65, 1023, 1024, 1025, 2047, 2048, 2049, 5000])
def test_row_lengths(nps, oracle, cuda_device, length):
    """Long rows at the lanes of a group where a run starts or ends, on a chain below them."""
    n = 6000
    rng = np.random.default_rng(length)
    heads = np.array([5504, 5505, 5530, 5535, 5536, 5568, 5599, 5999])
    s = [np.arange(1, 5504)] + [np.full(length, h) for h in heads]
    d = [np.arange(5503)] + [rng.integers(0, h, length) for h in heads]
    g = nps.convertCSR(n, np.concatenate(s), np.concatenate(d), np.ones(sum(x.size for x in s), np.uint32))
    _exact(nps, oracle, g)


@pytest.mark.parametrize("shape", [(1, 700), (700, 1), (33, 65), (300, 257)])
def test_grids(nps, oracle, cuda_device, shape):
    _exact(nps, oracle, nps.gen_grid(*shape, 0.05, 10, 3), threshold=7)


def test_malformed_rows_are_reported(nps, cuda_device):
    import torch
    g = nps.gen_uniform(5000, 40000, 10, 3)
    for at, value in ((77, -3), (77, 1 << 30), (4096, 5)):
        row = g.row_ptr.copy()
        row[at] = value
        t = [torch.from_numpy(a.view(np.int32)).to(cuda_device) for a in (row, g.col)]
        out = torch.empty(g.n, dtype=torch.int32, device=cuda_device)
        torch.cuda.synchronize()
        with pytest.raises(nps.NpsError) as ei:
            nps.color_device(*t, g.n, g.m, out)
        assert ei.value.status == 7
