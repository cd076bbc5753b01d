"""The root's training in one launch against the same steps on the CPU
(float64 gradient of oracle/mlp_oracle.py, Adam, projection): hidden sizes on
both sides of the padded widths, fewer samples than one CTA and more than all,
no step at all.  The reported losses are compared; 1e-3 of them covers FP32
sums over the samples through the steps taken."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _train(H, x, y, iters, lr):
    from oracle import mlp_oracle as mo
    p = np.concatenate([np.full(H, float(H)), -np.arange(H, dtype=float), np.full(H, 1.0 / H), [0.0]])
    m, v = np.zeros_like(p), np.zeros_like(p)
    losses = []
    for it in range(iters + 1):
        loss, g = mo.loss_grad(p, H, x, y)
        losses.append(loss)
        if it == iters:
            break
        m, v = 0.9 * m + 0.1 * g, 0.999 * v + 0.001 * g * g
        p = p - lr * (m / (1 - 0.9 ** (it + 1))) / (np.sqrt(v / (1 - 0.999 ** (it + 1))) + 1e-8)
        p[:H], p[2 * H:3 * H] = np.maximum(p[:H], 0), np.maximum(p[2 * H:3 * H], 0)
    return losses[0], losses[-1]


@pytest.mark.parametrize("H", [1, 15, 16, 17, 32])
@pytest.mark.parametrize("n,segs", [(5000, 40), (1 << 20, 60000)])
@pytest.mark.parametrize("iters", [0, 25])
def test_losses_follow_the_cpu_steps(bt, orc, cuda, H, n, segs, iters):
    import torch
    g = np.random.default_rng(n)
    keys = np.cumsum(np.floor(g.lognormal(4.0, 2.0, size=n)).astype(np.uint64) + 1)
    with bt.Tree.build(torch.from_numpy(keys).to(cuda), torch.arange(n, device=cuda)) as t:
        rep = t.learned_train(num_segments=segs, hidden=H, iterations=iters, learning_rate=0.002)
    starts, _, _ = orc.pla_segments(keys, rep["max_error"], chunk=1 << 14, hull_cap=32)
    first = keys[starts[::4].astype(np.int64)]  # first key of every segment line
    x = ((first - keys[0]).astype(np.float32) * np.float32(1.0 / float(keys[-1] - keys[0])))
    y = ((np.arange(len(first)) + 0.5) / len(first)).astype(np.float32)
    l0, l1 = _train(H, x, y, iters, 0.002)
    assert abs(rep["root_loss_initial"] - l0) <= 1e-3 * l0
    assert abs(rep["root_loss_final"] - l1) <= 1e-3 * l1
