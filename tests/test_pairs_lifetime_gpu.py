"""persistence_pairs returns while its last kernel reads the image again: the
image's memory must not go to another stream's tensors before that."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(120, 97), (3, 120, 97)])
def test_image_freed_right_after_the_call(monkeypatch, shape):
    from dmsc_b200 import autograd

    gen = torch.Generator(device="cuda").manual_seed(4)
    x = torch.rand(shape, generator=gen, device="cuda")
    ref = autograd.persistence_pairs(x, -1.0)
    extract = autograd._extract_raw

    def slow(*args):  # the pair kernel starts long after the call has returned
        r = extract(*args)
        torch.cuda._sleep(100_000_000)
        return r

    monkeypatch.setattr(autograd, "_extract_raw", slow)
    s = torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(s):
        q = autograd.persistence_pairs(x, -1.0)
    del x
    others = [torch.zeros(shape, device="cuda") for _ in range(16)]
    torch.cuda.synchronize()
    assert all(not o.any() for o in others)
    assert torch.equal(q.plus_pixel, ref.plus_pixel) and torch.equal(q.minus_pixel, ref.minus_pixel)
    assert torch.equal(q.persistence, ref.persistence)
