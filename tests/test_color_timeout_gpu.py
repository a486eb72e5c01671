"""nps_color's bounded waits: timeout_s bounds a wait in which nothing moves, not the chain
of colors before it.  On a path in id order some 75,000 vertices are in flight and the last
of them waits for all others, far longer than the timeout, while every vertex in turn gets
its color at once; a color that never comes still ends the call."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [3000, 80000, 200000])
def test_a_long_chain_outlasts_the_timeout(nps, oracle, cuda_device, n):
    g = nps.convertCSR(n, np.arange(1, n), np.arange(n - 1), np.ones(n - 1, np.uint32))
    got, st = nps.color(g, nps.Params(timeout_s=0.002))
    assert st.status == 0 and np.array_equal(got, 1 + np.arange(n)) and st.iterations == n


def test_a_color_that_never_comes_ends_the_call(nps, cuda_device):
    n = 80000
    g = nps.convertCSR(n, np.arange(1, n), np.arange(n - 1), np.ones(n - 1, np.uint32))
    with pytest.raises(nps.NpsError) as ei:
        nps.color(g, nps.Params(timeout_s=0.05, fault_inject_wait=True))
    assert ei.value.status == 4
    got, _ = nps.color(g)
    assert np.array_equal(got, 1 + np.arange(n))
