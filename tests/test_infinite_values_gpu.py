"""Infinite pixels under finite thresholds and an infinite threshold on finite
fields, against the oracle: the persistence of two equal infinities is NaN and
is never cancelled, and every finite pair is cancelled at threshold infinity.
(Both together are not compared: the thresholded roots then depend on the
order of the reference's unions.)"""

import numpy as np
import pytest
import torch

from tests.helpers import diff_fields

pytestmark = pytest.mark.gpu

INF = float("inf")


def _field(H, W, kind):
    rng = np.random.default_rng(100 * H + W)
    v = rng.random((H, W)).astype(np.float32)
    u = rng.random((H, W))
    if kind in ("high", "both"):
        v[u < 0.3] = INF
    if kind in ("low", "both"):
        v[u > 0.7] = -INF
    return torch.from_numpy(v)


@pytest.mark.parametrize("is_dual", [False, True])
@pytest.mark.parametrize("kind,thr", [(k, t) for k in ("high", "low", "both") for t in (0.0, 0.3, 3.0e38)]
                         + [("finite", INF), ("finite", -INF)])
@pytest.mark.parametrize("H,W", [(40, 41), (131, 70)])
def test_against_oracle(H, W, kind, thr, is_dual, oracle_mod):
    from dmsc_b200 import extract_dmsc

    img = _field(H, W, kind)
    exp = oracle_mod.run(img, thr, True, is_dual, False, False, True, True)
    assert diff_fields(extract_dmsc(img.cuda(), thr, True, is_dual, False, False, True, True), exp) == []


@pytest.mark.parametrize("is_dual", [False, True])
@pytest.mark.parametrize("kind", ["high", "low", "both"])
def test_both_infinite_stays_in_range(kind, is_dual):
    from dmsc_b200 import compute_dmsc

    c = compute_dmsc(_field(131, 70, kind).cuda(), INF, is_dual=is_dual, trace_ridges=False, trace_valleys=False)
    for lab, pts in ((c.peaks, c.max_pts), (c.basins, c.min_pts)):
        assert int(lab.min()) >= -1 and int(lab.max()) < max(len(pts), 1)
    for e, pts in ((c.e_max, c.max_pts), (c.e_min, c.min_pts)):
        if e.numel():
            assert int(e.min()) >= 0 and int(e[:, 0].max()) < len(c.sad_pts) and int(e[:, 1].max()) < len(pts)
