"""nps_bc's backward pass over long rows, whose heads on the next level gather 64 edges at a
time, are summed 32 at a time and leave 0 to 31 for the next step: rows of several steps in
which every step finds another number of them, so that each count left over meets each
count found.  Bit for bit as the oracle's restatement of bc_cpu."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("seed", range(6))
def test_heads_left_over_between_steps(nps, oracle, cuda_device, seed):
    """Hubs behind a source; an edge of a hub leads to a head of its own or, as the off-level
    one, back to the source.  Heads have 0 to 6 heads of their own."""
    rng = np.random.default_rng(seed)
    hubs, steps = 24, 40
    s, d, nxt = [np.zeros(hubs, np.int64)], [1 + np.arange(hubs)], 1 + hubs
    for h in range(hubs):
        on = rng.random(64 * steps - h) < np.repeat(rng.random(steps), 64)[:64 * steps - h]
        k = int(on.sum())
        to = np.zeros(on.size, np.int64)
        to[on] = nxt + np.arange(k) % 300
        s.append(np.full(on.size, 1 + h))
        d.append(to)
    tails = nxt + 300 + np.arange(900)
    cnt = rng.integers(0, 7, 300)
    s.append(np.repeat(nxt + np.arange(300), cnt))
    d.append(rng.choice(tails, int(cnt.sum())))
    s, d = np.concatenate(s), np.concatenate(d)
    g = nps.convertCSR(nxt + 1200, s, d, np.ones(s.shape[0], np.uint32))
    src = np.array([0, 1, 5, 0])
    got, want = np.asarray(nps.bc(g, src)[0], np.float32), np.asarray(oracle.bc(g.row_ptr, g.col, src), np.float32)
    assert np.array_equal(got.view(np.uint32), want.view(np.uint32))
