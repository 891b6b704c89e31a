"""Scans of the row segments, flags and survivors at sizes around a scan tile
(4096 items) and of several tiles, bit for bit against the oracle."""

import numpy as np
import pytest
import torch

from tests.helpers import diff_fields

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H,W", [(4094, 2), (4095, 3), (4096, 1), (12288, 5), (1, 40), (133, 127)])
def test_against_oracle(H, W):
    from dmsc_b200 import extract_dmsc
    from oracle import oracle

    img = torch.from_numpy(np.random.default_rng(H).random((H, W)).astype(np.float32))
    got = extract_dmsc(img.cuda(), 0.0, False, False, True, True, True, True)
    assert diff_fields(got, oracle.run(img, 0.0, False, False, True, True, True, True)) == []


def test_growing_and_shrinking_calls():
    """The scan's state outlives a call: larger and smaller ones in turn."""
    from dmsc_b200 import extract_dmsc
    from oracle import oracle

    for H, W in ((20, 30), (300, 200), (7, 7), (500, 400), (300, 200)):
        img = torch.from_numpy(np.random.default_rng(H + W).random((H, W)).astype(np.float32))
        got = extract_dmsc(img.cuda(), 0.02, False, True, True, True, True, True)
        assert diff_fields(got, oracle.run(img, 0.02, False, True, True, True, True, True)) == []
