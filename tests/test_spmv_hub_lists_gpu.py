"""nps_spmv at the WARP and BLOCK levels in matrices of at least 2^19 nonzeros, where rows
from 2,048 nonzeros on are listed and take the grid level's chunks: rows around that length
and around chunks of 1,024, thresholds below and beyond it, matrices on both sides of 2^19
nonzeros, and overlapping rows, which hold more rows and chunks than the lists.  Which path
a long row took shows in its bits: a chunk's sum and a walk by one warp or CTA round
differently, and the grid level always takes the chunks."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
MIN_NNZ, HUB = 1 << 19, 2048
HUBS = np.array([0, 31, 32, 33, 20000, 33333])


def _matrix(nps, m, length, hubs=HUBS, cols=40000):
    """m nonzeros, the hub rows first drawn and so the same in every matrix of this length."""
    rng = np.random.default_rng(length)
    hub_cols = rng.integers(0, cols, (hubs.size, length))
    n = 250_000
    rest = m - hubs.size * length
    row = rng.integers(0, n - hubs.size, rest)
    free = np.setdiff1d(np.arange(n), hubs)
    s = np.concatenate([np.repeat(hubs, length), free[row]])
    d = np.concatenate([hub_cols.ravel(), rng.integers(0, n, rest)])
    g = nps.convertCSR(n, s, d, np.ones(m, np.uint32))
    assert g.m == m
    return g


@pytest.mark.parametrize("level", [0, 1])
@pytest.mark.parametrize("length", [2046, 2047, 2048, 2049, 3071, 3072, 3073, 40000])
def test_long_rows(nps, oracle, cuda_device, level, length):
    g = _matrix(nps, 700_000, length)
    val, x = oracle.spmv_data(g.n, g.m)
    want = oracle.spmv(g.row_ptr, g.col, val, x)  # exact in double, whatever the order
    for threshold in (32, 2047, 2048, 5000, 1 << 20):
        y, st = nps.spmv(g, val, x, nps.Params(level=level, threshold=threshold))
        assert st.status == 0 and np.array_equal(y, want)


@pytest.mark.parametrize("level", [0, 1])
@pytest.mark.parametrize("m", [MIN_NNZ - 1, MIN_NNZ, MIN_NNZ + 1])
@pytest.mark.parametrize("length", [HUB - 1, HUB, 5000])
def test_which_rows_take_chunks(nps, cuda_device, level, m, length):
    """40 hub rows of random values: the grid level's bits exactly where they take chunks."""
    hubs = np.arange(100, 40100, 1000)
    g = _matrix(nps, m, length, hubs)
    rng = np.random.default_rng(1)
    val, x = rng.standard_normal(g.m), rng.standard_normal(g.n)
    grid = nps.spmv(g, val, x, nps.Params(level=2, threshold=64))[0][hubs]
    y = nps.spmv(g, val, x, nps.Params(level=level, threshold=64))[0]
    ref = np.add.reduceat(np.append(val * x[g.col], 0.0), g.row_ptr[:-1]) * (np.diff(g.row_ptr) > 0)
    bound = np.add.reduceat(np.append(np.abs(val * x[g.col]), 0.0), g.row_ptr[:-1])
    assert np.all(np.abs(y - ref) <= 2 * length * np.finfo(np.float64).eps * bound + 1e-300)
    if m >= MIN_NNZ and length >= HUB:
        assert np.array_equal(y[hubs], grid)
    else:
        assert not np.array_equal(y[hubs], grid)


@pytest.mark.parametrize("level", [0, 1])
def test_overlapping_rows_are_reported(nps, cuda_device, level):
    """2,000 rows that claim the whole matrix, where the lists hold about 300."""
    import torch
    n = 4000
    g = nps.gen_uniform(n, 600_000, 10, 3)
    assert g.m >= MIN_NNZ and g.m // HUB + 1 < n // 2
    row = g.row_ptr.copy()
    row[1:n:2] = g.m
    row[0:n:2] = 0
    t = [torch.from_numpy(a.view(np.int32)).to(cuda_device) for a in (row, g.col)]
    val, x = (torch.ones(k, dtype=torch.float64, device=cuda_device) for k in (g.m, g.n))
    y = torch.empty(g.n, dtype=torch.float64, device=cuda_device)
    torch.cuda.synchronize()
    with pytest.raises(nps.NpsError) as ei:
        nps.spmv_device(*t, val, x, y, g.n, g.m, nps.Params(level=level, threshold=16))
    assert ei.value.status == 7
