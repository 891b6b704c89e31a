"""V-paths that cross the border between two label tiles many times."""

import numpy as np
import pytest
import torch

from tests.helpers import diff_fields

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dual", [False, True])
def test_path_crosses_a_tile_border_often(dual):
    """62 x 64 pixels: the index grid has two label tiles, the second one
    column wide; on this field of four values a path crosses their border more
    often than there are tiles."""
    from dmsc_b200 import extract_dmsc
    from oracle import oracle

    img = torch.from_numpy(np.floor(4 * np.random.default_rng(62064).random((62, 64))).astype(np.float32))
    got = extract_dmsc(img.cuda(), 0.1, True, dual, True, True, True, True)
    assert diff_fields(got, oracle.run(img, 0.1, True, dual, True, True, True, True)) == []


def _field(kind, H, W):
    """'snake': one ramp through the rows in turn, down a row at a time, so a
    path visits every cell of a tile; 'ties': four values; 'noise'."""
    if kind == "snake":
        y, x = np.mgrid[0:H, 0:W]
        ramp = y * (W + 2) + np.where(y & 1, W - x, x)
        return np.where((y & 1) & ((x != np.where(y & 2, 0, W - 1))), 1e6 + ramp, ramp).astype(np.float32)
    r = np.random.default_rng(H * 1000 + W).random((H, W))
    return (np.floor(4 * r) if kind == "ties" else r).astype(np.float32)


@pytest.mark.parametrize("kind", ["snake", "ties", "noise"])
@pytest.mark.parametrize("H,W", [(2, 2), (31, 33), (63, 64), (64, 63), (65, 129), (126, 62), (3, 190), (190, 3)])
def test_tile_edges(H, W, kind):
    """Sizes around the 64 x 64 label tiles, both sides and either alone."""
    from dmsc_b200 import extract_dmsc
    from oracle import oracle

    img = torch.from_numpy(_field(kind, H, W))
    for dual, peaks, basins in ((False, True, True), (True, True, False), (False, False, True)):
        args = (0.0, True, dual, False, False, peaks, basins)
        assert diff_fields(extract_dmsc(img.cuda(), *args), oracle.run(img, *args)) == []
