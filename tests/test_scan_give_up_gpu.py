"""A scan whose tiles do not find their predecessors' sums ends the call with
an error before anything is addressed by its output, and the context stays
usable."""

import pytest
import torch

from tests.helpers import diff_fields

pytestmark = pytest.mark.gpu


# (H, W, launches up to the failure): 4096 row segments of 32 indices make a
# tile, so the first size has one tile in the first scan (row segments) and
# several in the second (flags), where the pairing has run; the others have
# several in the first, after the gradient kernel and nothing else
@pytest.mark.parametrize("H,W,launches", [(256, 256, None), (1024, 1024, 2), (2048, 1001, 2)])
def test_scan_that_gives_up(H, W, launches):
    from dmsc_b200 import _lib, compute_dmsc

    img = torch.rand(H, W, generator=torch.Generator().manual_seed(H + W)).cuda()
    ref = compute_dmsc(img, 0.01)
    ctx = _lib.context(torch.cuda.current_device())
    try:
        ctx.set_scan_looks(-1)
        with pytest.raises(RuntimeError, match="bounded device loop reached its cap"):
            compute_dmsc(img, 0.01)
        if launches is not None:
            assert ctx.launch_count() == launches
    finally:
        ctx.set_scan_looks()
    assert diff_fields(compute_dmsc(img, 0.01), ref) == []


def test_scan_of_one_tile_looks_for_nothing():
    from dmsc_b200 import _lib, compute_dmsc

    img = torch.rand(20, 31, generator=torch.Generator().manual_seed(1)).cuda()
    ref = compute_dmsc(img, 0.01)
    ctx = _lib.context(torch.cuda.current_device())
    try:
        ctx.set_scan_looks(-1)
        assert diff_fields(compute_dmsc(img, 0.01), ref) == []
    finally:
        ctx.set_scan_looks()
