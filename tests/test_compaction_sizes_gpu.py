"""Critical-cell lists at the edges of the compaction's work split (warps of
8 consecutive 32-column row segments, lists handled 32 entries at a time)."""

import numpy as np
import pytest
import torch

from tests.helpers import diff_fields

pytestmark = pytest.mark.gpu


def _field(kind, H, W):
    y, x = np.mgrid[0:H, 0:W]
    noise = np.random.default_rng(H * 1000 + W).random((H, W))
    if kind == "checker":  # as many critical cells as a field can have
        return ((y + x) % 2 + 0.25 * noise).astype(np.float32)
    if kind == "ramp":  # almost none
        return (y * W + x).astype(np.float32)
    v = noise.astype(np.float32)
    v[noise < 0.1] = -0.0
    v[noise > 0.9] = np.inf
    return v


@pytest.mark.parametrize("kind", ["checker", "ramp", "noise"])
@pytest.mark.parametrize("H,W", [(1, 1), (1, 300), (300, 1), (7, 31), (7, 32), (8, 63), (15, 255), (16, 256), (64, 130)])
def test_lists_match_the_oracle(H, W, kind):
    from dmsc_b200 import extract_dmsc
    from oracle import oracle

    img = torch.from_numpy(_field(kind, H, W))
    for dual in (False, True):
        args = (0.0, True, dual, True, True, True, True)
        want = oracle.run(img, *args)
        assert diff_fields(extract_dmsc(img.cuda(), *args), want) == []
        for got in extract_dmsc(torch.stack([img, img, img]).cuda(), *args):  # segments of several images in a warp
            assert diff_fields(got, want) == []
