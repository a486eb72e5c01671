"""nps_bc on graphs whose levels reach the reference's mark of unvisited vertices (9999):
paths around that length, in one and in both directions, below and above the vertex count
up to which a source fits shared memory, from one source and from several (some of them
shallow).  Bit for bit as the oracle's restatement of bc_cpu.  A vertex on level 9999 that
is taken more often than there is room for ends the call with an error.  And calls of many
sources on graphs of many small levels, which change the kernel on the way."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _same(a, b):
    """Bit for bit, NaNs (0 / 0 where path counts wrap) as NaNs."""
    a, b = np.asarray(a, np.float32), np.asarray(b, np.float32)
    return bool(np.all((a.view(np.uint32) == b.view(np.uint32)) | (np.isnan(a) & np.isnan(b))))


def _path(nps, n, both):
    a, b = np.arange(n - 1), np.arange(1, n)
    s, d = (np.concatenate([a, b]), np.concatenate([b, a])) if both else (a, b)
    return nps.convertCSR(n, s, d, np.ones(s.shape[0], np.uint32))


@pytest.mark.parametrize("n", [9998, 9999, 10000, 10001, 10002, 12000, 17600, 18500])
@pytest.mark.parametrize("both", [False, True])
def test_paths(nps, oracle, cuda_device, n, both):
    g = _path(nps, n, both)
    for src in ([0], [n // 2, n - 1, 0, 7] + list(range(20, 400, 2))):
        got, st = nps.bc(g, np.array(src))
        assert st.status == 0 and _same(got, oracle.bc(g.row_ptr, g.col, src))


@pytest.mark.parametrize("n,k", [(10100, 5000), (20000, 15000)])
def test_repeated_visits_end_with_an_error(nps, oracle, cuda_device, n, k):
    """k edges from level 9998 to one vertex, where n + 4,096 - 9,999 visits have room; the
    library works on afterwards."""
    s = np.concatenate([np.arange(9998), np.full(k, 9998)])
    d = np.concatenate([np.arange(1, 9999), np.full(k, 9999)])
    g = nps.convertCSR(n, s, d, np.ones(s.shape[0], np.uint32))
    with pytest.raises(nps.NpsError) as ei:
        nps.bc(g, np.array([0]))
    assert ei.value.status == 3
    got, st = nps.bc(g, np.array([1]))  # one level less: every edge counts
    assert st.status == 0 and _same(got, oracle.bc(g.row_ptr, g.col, [1]))


@pytest.mark.parametrize("shape,sources", [((64, 64), 0), ((3, 700), 0), ((90, 100), 500), ((17, 17), 0)])
def test_many_sources_on_grids(nps, oracle, cuda_device, shape, sources):
    g = nps.gen_grid(*shape, 0.05, 10, 5)
    src = None if sources == 0 else np.linspace(0, g.n - 1, sources).astype(np.int64)
    for block in (0, 7, 333):  # sources per block of dependency rows
        got, st = nps.bc(g, src, nps.Params(bc_block_sources=block))
        assert st.status == 0 and _same(got, oracle.bc(g.row_ptr, g.col, src))


@pytest.mark.parametrize("n,ctas_per_sm", [(17650, 1), (17651, 8)])
def test_the_shared_memory_limit(nps, oracle, cuda_device, n, ctas_per_sm):
    """The largest vertex count of the shared-memory kernel (one CTA per SM there) and the next."""
    import torch
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    g = nps.gen_uniform(n, 4 * n, 10, n)
    src = np.arange(2 * sms)
    got, st = nps.bc(g, src)
    assert st.status == 0 and _same(got, oracle.bc(g.row_ptr, g.col, src))
    assert st.grid_ctas == min(ctas_per_sm, 2) * sms


@pytest.mark.parametrize("share", [0.05, 0.2, 0.3, 0.9])
def test_part_of_the_sources_on_a_chain(nps, oracle, cuda_device, share):
    """A power-law graph and a chain beside it: which kernel ends the call depends on how many
    of the first sources lie on the chain, the result does not."""
    core = nps.gen_rmat(11, 8, seed=3)
    ln = 3000
    s = np.concatenate([np.repeat(np.arange(core.n), core.degrees()), core.n + np.arange(ln - 1)])
    d = np.concatenate([core.col, core.n + 1 + np.arange(ln - 1)])
    g = nps.convertCSR(core.n + ln, s, d, np.ones(s.shape[0], np.uint32))
    rng = np.random.default_rng(7)
    src = np.where(rng.random(2500) < share, core.n + rng.integers(0, ln, 2500), rng.integers(0, core.n, 2500))
    got, st = nps.bc(g, src)
    assert st.status == 0 and _same(got, oracle.bc(g.row_ptr, g.col, src))
