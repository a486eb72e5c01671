"""nps_spmv at the WARP and BLOCK levels around the row length (2,048 nonzeros) from which
rows take the grid level's chunks, next to chunk boundaries, and at thresholds beyond it;
and row offsets whose rows overlap, which hold more rows and chunks than the lists.  With
the reference's data every sum is exact in double, so y equals the oracle's bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("level", [0, 1, 2])
@pytest.mark.parametrize("length", [2046, 2047, 2048, 2049, 3071, 3072, 3073, 40000])
def test_long_rows(nps, oracle, cuda_device, level, length):
    n = 50000
    rng = np.random.default_rng(length)
    lens = rng.integers(0, 6, n)
    lens[[0, 31, 32, 33, 20000, n - 1]] = length
    src = np.repeat(np.arange(n), lens)
    g = nps.convertCSR(n, src, rng.integers(0, n, src.shape[0]), np.ones(src.shape[0], np.uint32))
    val, x = oracle.spmv_data(g.n, g.m)
    want = oracle.spmv(g.row_ptr, g.col, val, x)
    for threshold in (32, 2048, 5000, 1 << 20):
        y, st = nps.spmv(g, val, x, nps.Params(level=level, threshold=threshold))
        assert st.status == 0 and np.array_equal(y, want)


@pytest.mark.parametrize("level", [0, 1, 2])
def test_overlapping_rows_are_reported(nps, cuda_device, level):
    import torch
    g = nps.gen_uniform(4000, 40000, 10, 3)
    row = g.row_ptr.copy()
    row[1:4000:2] = g.m  # every other row claims the whole matrix, the ones between run backwards
    row[0:4000:2] = 0
    t = [torch.from_numpy(a.view(np.int32)).to(cuda_device) for a in (row, g.col)]
    val, x = (torch.ones(k, dtype=torch.float64, device=cuda_device) for k in (g.m, g.n))
    y = torch.empty(g.n, dtype=torch.float64, device=cuda_device)
    torch.cuda.synchronize()
    with pytest.raises(nps.NpsError) as ei:
        nps.spmv_device(*t, val, x, y, g.n, g.m, nps.Params(level=level, threshold=16))
    assert ei.value.status == 7
