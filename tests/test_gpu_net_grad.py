"""The network's gradients where the gathering of a set's points can go wrong: every channel on one point, as many points as
there are, one sample, and more sets than the launch has CTAs."""

import numpy as np
import pytest
import torch

from oracle import oracle

pytestmark = pytest.mark.gpu


def _sets(kind, n, rng):
    x = np.zeros((2 * n, 1024, 4), np.float32)
    if kind == "same":  # one point 1024 times: the argmax is the first for every channel
        x[..., :3] = rng.uniform(-4.0, 4.0, (2 * n, 1, 3))
    elif kind == "shell":  # far points in every direction: many distinct argmax points
        d = rng.normal(0.0, 1.0, (2 * n, 1024, 3))
        x[..., :3] = 8.0 * d / np.linalg.norm(d, axis=2, keepdims=True)
    else:
        x[..., :3] = rng.uniform(-5.0, 5.0, (2 * n, 1024, 3))
    return x


def _net(n):
    from livox_warp.initnet import InitNet

    return InitNet(seed=5, batch_cap=n)


@pytest.mark.parametrize("kind,n", [("same", 1), ("same", 3), ("shell", 2), ("box", 3)])
def test_gradient_against_the_oracle(kind, n):
    rng = np.random.default_rng(11)
    net = _net(n)
    x = _sets(kind, n, rng)
    tgt = rng.normal(0.0, 0.05, (n, 6))
    sets = torch.from_numpy(x).cuda()
    fwd = net.forward(sets, n)
    net.backward(sets, n, fwd, torch.from_numpy(tgt).float())
    got = net.grad.cpu().numpy().astype(np.float64)
    w = net.w.cpu().numpy().view(np.uint16)
    ref = oracle.net_forward(w, x, net.in_scale, net.out_scale.cpu().numpy())
    # the same argmax points on both sides (a near tie may go either way): the device's
    ref["argmax"] = fwd["argmax"].cpu().numpy().reshape(2 * n, 256)
    want, _ = oracle.net_backward(w, x, ref, tgt.astype(np.float32), np.ones(6), net.out_scale.cpu().numpy())
    for o, size in ((0, 192), (192, 64), (256, 8192), (8448, 128), (8576, 32768), (41344, 256)):
        a, b = got[o:o + size], want[o:o + size]
        assert np.linalg.norm(a - b) <= 0.02 * np.linalg.norm(b) + 1e-7  # the bf16 activations' bound (test_gpu_initnet)


@pytest.mark.parametrize("n", [1, 74, 149, 333])
def test_gradient_is_the_samples_sum(n):
    """Losses and gradients are means over the samples: a batch's gradient is the mean of its samples' own, whatever CTA
    they fall to. Sums of n float32 terms in another order: 4 (log2 n + 24) 2^-24 of the norm is ample."""
    rng = np.random.default_rng(12)
    net = _net(n)
    sets = torch.from_numpy(_sets("box", n, rng)).cuda()
    tgt = torch.from_numpy(rng.normal(0.0, 0.05, (n, 6))).float().cuda()
    fwd = net.forward(sets, n)
    loss = float(net.backward(sets, n, fwd, tgt).sum())
    got = net.grad.double().clone()
    one = _net(1)
    total, losses = torch.zeros_like(got), 0.0
    for k in range(n):
        s = sets[2 * k:2 * k + 2].contiguous()
        f = one.forward(s, 1)
        losses += float(one.backward(s, 1, f, tgt[k:k + 1]).sum()) / n
        total += one.grad.double() / n
    bound = 4.0 * (np.log2(n) + 24) * 2.0 ** -24
    assert abs(loss - losses) <= bound * abs(losses)
    assert float((got - total).norm()) <= bound * float(total.norm())
