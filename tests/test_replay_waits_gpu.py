"""Replay of long chains of cancellations, where most walks wait for decisions
made in the same round: smooth fields in few levels (ties in value and in
persistence) and nested slopes, bit for bit against the oracle."""

import numpy as np
import pytest
import torch

from tests.helpers import diff_fields

pytestmark = pytest.mark.gpu


def _field(kind, H, W):
    rng = np.random.default_rng(7 * H + W)
    y, x = np.mgrid[0:H, 0:W]
    a = np.sin(x / 11.0) + np.cos(y / 13.0) + 0.3 * np.sin((x + 2 * y) / 3.0)
    if kind == "levels":
        a = np.round(12 * (a + 0.05 * rng.standard_normal((H, W)))) / 12
    elif kind == "slope":  # persistences grow along the slope: deep parent chains
        a = 0.01 * x + (0.02 + 0.0004 * x) * rng.random((H, W))
    else:
        a = a + 0.2 * rng.standard_normal((H, W))
    return torch.from_numpy(a.astype(np.float32))


@pytest.mark.parametrize("dual", [False, True])
@pytest.mark.parametrize("kind", ["levels", "slope", "noise"])
@pytest.mark.parametrize("H,W,thr", [(33, 700, 0.3), (200, 201, 0.5), (1, 300, 0.2)])
def test_against_oracle(H, W, thr, kind, dual):
    from dmsc_b200 import extract_dmsc
    from oracle import oracle

    img = _field(kind, H, W)
    got = extract_dmsc(img.cuda(), thr, False, dual, True, True, True, True)
    assert diff_fields(got, oracle.run(img, thr, False, dual, True, True, True, True)) == []
