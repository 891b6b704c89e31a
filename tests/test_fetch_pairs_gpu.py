"""Entries of ``persistence_pairs`` against the oracle's p and pair lists, for
the smallest images, odd sizes and batches of mixed orientation."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("thr", [-1.0, 0.1])
@pytest.mark.parametrize("B,H,W", [(1, 1, 1), (1, 1, 9), (3, 7, 1), (2, 65, 64), (5, 33, 70)])
def test_entries_against_oracle(B, H, W, thr):
    from dmsc_b200.autograd import persistence_pairs
    from oracle import oracle

    rng = np.random.default_rng(100 * H + W)
    x = torch.from_numpy(rng.random((B, H, W)).astype(np.float32))
    duals = [bool(b % 2) for b in range(B)]
    q = persistence_pairs(x.cuda().requires_grad_(), thr, duals)
    p, image, side, ppairs, plus, minus = (t.detach().cpu() for t in (
        q.persistence, q.image, q.side, q.ppairs, q.plus_pixel, q.minus_pixel))
    at = 0
    for b in range(B):
        out = oracle.run(x[b], thr, False, duals[b], False, False, False, False)
        p_max, p_min, pp_max, pp_min = out[6], out[7], out[8], out[9]
        n = p_min.numel()
        e = slice(at, at + 2 * n)
        assert torch.equal(p[e], torch.cat([p_min, p_max]))
        assert torch.equal(ppairs[e], torch.cat([pp_min, pp_max]))
        assert torch.equal(image[e], torch.full((2 * n,), b)) and image.dtype == torch.int64
        assert side[e].tolist() == [0] * n + [1] * n and side.dtype == torch.int8
        v = x[b].reshape(-1)
        real = plus[e] >= 0
        assert torch.equal(real, p[e] != -1.0) and torch.equal(real, minus[e] >= 0)
        assert torch.equal(v[plus[e][real].long()] - v[minus[e][real].long()], p[e][real])
        at += 2 * n
    assert at == p.numel()


def test_backward_reaches_each_image():
    from dmsc_b200.autograd import persistence_pairs

    rng = np.random.default_rng(3)
    x = torch.from_numpy(rng.random((3, 40, 31)).astype(np.float32)).cuda().requires_grad_()
    q = persistence_pairs(x, -1.0, [False, True, False])
    w = torch.arange(1, q.persistence.numel() + 1, device="cuda", dtype=torch.float32)
    (q.persistence * w).sum().backward()
    exp = torch.zeros(3, 40 * 31, dtype=torch.float64)
    for e in range(w.numel()):
        if int(q.plus_pixel[e]) >= 0:
            exp[int(q.image[e]), int(q.plus_pixel[e])] += float(w[e])
            exp[int(q.image[e]), int(q.minus_pixel[e])] -= float(w[e])
    # sums of a few whole numbers below 2^24: exact
    assert torch.equal(x.grad.reshape(3, -1).double().cpu(), exp)
