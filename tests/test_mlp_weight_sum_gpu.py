"""The weighted mean of nps_mlp_loss_backward around the batch size (32,768) where the sum
of the sample weights moves from the loss kernel's CTAs to a kernel of its own, and at
batches around a warp and a CTA.  Against float64 autograd on the bf16-rounded matrices.

Tolerance, per gradient element: 1e-4 of the sum of its terms' magnitudes.  A term takes
fewer than 100 float roundings (dot products of 12 and 32, two exponentials, the products
of the chain rule): 6e-6.  The sum over the batch passes a 5-step tree, at most 8 additions
per CTA accumulator and at most 1,184 atomic additions: 1,200 roundings, 7.2e-5."""
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("weighted", [True, False])
@pytest.mark.parametrize("batch", [1, 31, 33, 127, 129, 1025, 32767, 32768, 32769])
def test_gradients_match_float64(nps, cuda_device, batch, weighted):
    import torch
    pol = importlib.import_module("nested-parallelism_b200.policy")
    r = np.random.default_rng(batch)
    x = r.standard_normal((batch, pol.IN)).astype(np.float32)
    yd = np.where(r.random(batch) < 0.5, r.integers(0, pol.N_DELTA, batch), -1).astype(np.int32)
    yl = r.integers(0, pol.N_LEVEL, batch).astype(np.int32)
    wt = r.uniform(0.1, 4.0, batch).astype(np.float32)
    w = pol.MLPWeights.init(batch)
    tr = pol.GPUTrainer(w, cuda_device)
    dev = [torch.from_numpy(a).to(cuda_device) for a in (x, yd, yl, wt)]
    torch.cuda.synchronize()
    for _ in range(2):  # the second call must not see the first one's sums
        loss = float(tr.loss_backward(dev[0], dev[1], dev[2], dev[3] if weighted else None).item())
    got = [g.double().cpu().numpy() for g in tr.grad]

    w1, w2 = pol.bf16_round(w.w1).astype(np.float64), pol.bf16_round(w.w2).astype(np.float64)
    h = np.maximum(x.astype(np.float64) @ w1.T + w.b1, 0.0)
    o = h @ w2.T + w.b2
    sc = wt.astype(np.float64) / wt.astype(np.float64).sum() if weighted else np.full(batch, 1.0 / batch)
    d, want = np.zeros_like(o), 0.0
    for lo, hi, y in ((0, pol.N_DELTA, yd), (pol.N_DELTA, pol.OUT, yl)):
        z = o[:, lo:hi] - o[:, lo:hi].max(1, keepdims=True)
        p = np.exp(z) / np.exp(z).sum(1, keepdims=True)
        has = y >= 0
        hot = np.zeros_like(p)
        hot[has, y[has]] = 1.0
        d[:, lo:hi] = np.where(has[:, None], sc[:, None] * (p - hot), 0.0)
        want += -(sc[has] * np.log(p[has, y[has]])).sum()
    dh = (d @ w2) * (h > 0)
    ax, ah, ad, adh = np.abs(x).astype(np.float64), h, np.abs(d), np.abs(d) @ np.abs(w2) * (h > 0)
    refs = [(dh.T @ x.astype(np.float64), adh.T @ ax), (dh.sum(0), adh.sum(0)), (d.T @ h, ad.T @ ah),
            (d.sum(0), ad.sum(0))]
    assert abs(loss - want) <= 1e-4 * abs(want)
    for g, (ref, mag) in zip(got, refs):
        assert np.all(np.abs(g - ref) <= 1e-4 * mag + 1e-30)
