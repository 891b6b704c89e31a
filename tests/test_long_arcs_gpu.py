"""Raw arcs of more cells than a survivor's record holds (15 bits a length),
and the fetch in two halves."""

import ctypes

import numpy as np
import pytest
import torch

from tests.helpers import diff_fields

pytestmark = pytest.mark.gpu


def _corridor(S):
    """One rising corridor winding through an S x S field between high walls."""
    img = np.full((S, S), -1.0)
    k = 0
    for y in range(0, S, 2):
        right = (y // 2) % 2 == 0
        for x in range(S) if right else range(S - 1, -1, -1):
            img[y, x] = k
            k += 1
        if y + 2 < S:
            img[y + 1, S - 1 if right else 0] = k
            k += 1
    wall = img < 0
    img[wall] = 2 * S * S + np.arange(wall.sum())
    return torch.from_numpy(img.astype(np.float32))


@pytest.mark.parametrize("S", [254, 256, 300])
def test_corridor(S):
    """Arcs of up to about S^2 / 2 cells: 32 512, 33 023 and 45 300, around and above 2^15 - 1."""
    from dmsc_b200 import extract_dmsc
    from oracle import oracle

    for img, dual in ((_corridor(S), False), (-_corridor(S), True)):
        args = (0.0, True, dual, True, True, True, True)
        assert diff_fields(extract_dmsc(img.cuda(), *args), oracle.run(img, *args)) == []


def test_fetch_finish_needs_a_start():
    from dmsc_b200 import _lib, compute_dmsc

    img = _corridor(20).cuda()
    compute_dmsc(img, 0.0)
    ctx = _lib.context(torch.cuda.current_device())
    rc = ctx.lib.dmsc_b200_fetch_finish(ctx.h, ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    with pytest.raises(RuntimeError, match="fetch_finish without a fetch_start"):
        ctx.check(rc, "dmsc_b200_fetch_finish")
    compute_dmsc(img, 0.0)  # the context stays usable
