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
