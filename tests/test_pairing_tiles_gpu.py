"""The pairing's tile pass and its hand-over to the grid's and the last block's
rounds: sizes around the 64 x 64 tiles, tiles with more extrema or saddles
than fit in shared memory next to tiles that do, paths that leave their tile,
and ties, every output bit for bit against the oracle."""

import numpy as np
import pytest
import torch

from tests.helpers import diff_fields

pytestmark = pytest.mark.gpu


def _field(kind, H, W):
    rng = np.random.default_rng(1000 * H + W)
    y, x = np.mgrid[0:H, 0:W]
    a = rng.random((H, W))
    if kind == "dense":  # every second pixel a minimum: no tile fits
        a = ((x + y) & 1) + 0.4 * a
    elif kind == "mixed":  # dense columns beside smooth ones
        a = np.where((x // 64) % 2 == 0, ((x + y) & 1) + 0.4 * a, np.sin(x / 9.0) + np.cos(y / 7.0) + 0.1 * a)
    elif kind == "ramp":  # long paths: most extrema lie in another tile than their saddles
        a = 0.05 * x + 0.02 * y + 0.06 * a
    elif kind == "ties":
        a = np.floor(4 * a)
    return torch.from_numpy(a.astype(np.float32))


@pytest.mark.parametrize("dual", [False, True])
@pytest.mark.parametrize("kind", ["noise", "dense", "mixed", "ramp", "ties"])
@pytest.mark.parametrize("H,W", [(63, 63), (62, 64), (64, 129), (1, 200), (130, 1), (191, 257)])
def test_against_oracle(H, W, kind, dual):
    from dmsc_b200 import extract_dmsc
    from oracle import oracle

    img = _field(kind, H, W)
    got = extract_dmsc(img.cuda(), 0.1, True, dual, True, True, True, True)
    assert diff_fields(got, oracle.run(img, 0.1, True, dual, True, True, True, True)) == []


@pytest.mark.parametrize("kind", ["noise", "dense"])
def test_grid_rounds_against_oracle(kind):
    """Enough undecided saddles that the grid's rounds run before the last block's."""
    from dmsc_b200 import extract_dmsc
    from oracle import oracle

    img = _field(kind, 450, 700)
    got = extract_dmsc(img.cuda(), 0.0, False, False, False, False, True, True)
    assert diff_fields(got, oracle.run(img, 0.0, False, False, False, False, True, True)) == []
