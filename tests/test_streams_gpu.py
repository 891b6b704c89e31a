"""Calls of one thread on several streams: a call that returns while its
kernels still read the context's buffers must not be overtaken by the next
one. Each case is compared with the same calls made one after the other."""

import ctypes

import numpy as np
import pytest
import torch

from tests.helpers import diff_fields

pytestmark = pytest.mark.gpu

DELAY = 100_000_000  # clock cycles, about 50 ms


def _fields(shape, seed):
    rng = np.random.default_rng(seed)
    return torch.from_numpy(rng.random(shape).astype(np.float32)).cuda()


def _same_pairs(q, ref):
    for name in ("persistence", "image", "side", "ppairs", "plus_pixel", "minus_pixel"):
        assert torch.equal(getattr(q, name), getattr(ref, name)), name


@pytest.mark.parametrize("delayed", [False, True])
def test_pairs_then_a_call_on_another_stream(monkeypatch, delayed):
    from dmsc_b200 import autograd, compute_dmsc

    x, y = _fields((8, 257, 300), 1), _fields((700, 333), 2)
    duals = [b % 2 == 1 for b in range(8)]
    ref_q, ref_c = autograd.persistence_pairs(x, -1.0, duals), compute_dmsc(y, 0.02)
    extract = autograd._extract_raw

    def slow(*args):  # the pair kernel starts long after the next call has been made
        r = extract(*args)
        torch.cuda._sleep(DELAY)
        return r

    if delayed:
        monkeypatch.setattr(autograd, "_extract_raw", slow)
    s1, s2 = torch.cuda.Stream(), torch.cuda.Stream()
    torch.cuda.synchronize()
    for _ in range(3):
        with torch.cuda.stream(s1):
            q = autograd.persistence_pairs(x, -1.0, duals)
        with torch.cuda.stream(s2):
            c = compute_dmsc(y, 0.02)
        torch.cuda.synchronize()
        _same_pairs(q, ref_q)
        assert diff_fields(c, ref_c) == []


def test_backward_on_two_streams():
    from dmsc_b200.autograd import persistence_pairs, scatter_pair_grads

    terms = []
    for B, seed in ((16, 3), (3, 4)):
        q = persistence_pairs(_fields((B, 256, 256), seed), -1.0)
        n = 256 * 256
        flat = [torch.where(p >= 0, p + (q.image * n).int(), p) for p in (q.plus_pixel, q.minus_pixel)]
        terms.append((*flat, q.persistence, (B, 256, 256)))
    ref = [scatter_pair_grads(*t) for t in terms]
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    for _ in range(3):
        out = []
        for s, t in zip(streams, terms):
            with torch.cuda.stream(s):
                out.append(scatter_pair_grads(*t))
        torch.cuda.synchronize()
        assert all(torch.equal(a, b) for a, b in zip(out, ref))


def test_backward_under_capture():
    """The events that order calls on different streams stay out of a capture."""
    from dmsc_b200.autograd import persistence_pairs, scatter_pair_grads

    q = persistence_pairs(_fields((64, 80), 5), -1.0)
    ref = scatter_pair_grads(q.plus_pixel, q.minus_pixel, q.persistence, (64, 80))
    g = torch.zeros_like(q.persistence)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = scatter_pair_grads(q.plus_pixel, q.minus_pixel, g, (64, 80))
    g.copy_(q.persistence)
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(out, ref)


class _Raw:
    """The two phases of one image through the C ABI, each on a stream of its
    own, into buffers like the fields of ``ref``."""

    def __init__(self, img, thr, ref):
        from dmsc_b200 import _lib
        from dmsc_b200.dmsc import _FIELDS

        self.lib, self.L, self.img, self.thr, self.ref = _lib.load(), _lib, img, thr, ref
        self.ctx = _lib.context(torch.cuda.current_device())
        self.out = {f: torch.empty_like(getattr(ref, f)) for f in (*_FIELDS, "grad_indices", "peaks", "basins")}
        self.ptr = {f: ctypes.c_void_p(t.data_ptr()) for f, t in self.out.items()}
        self.outputs = _lib.Outputs(**{f: self.ptr[f] for f in _FIELDS})
        torch.cuda.synchronize()

    def extract(self, stream):
        L, (H, W) = self.L, self.img.shape
        flags = L.RETURN_GRADIENT | L.TRACE_RIDGES | L.TRACE_VALLEYS | L.TRACE_PEAKS | L.TRACE_BASINS
        sizes = L.Sizes()
        rc = self.lib.dmsc_b200_extract(self.ctx.h, ctypes.c_void_p(self.img.data_ptr()), H, W,
                                        ctypes.c_float(self.thr), flags, self.ptr["grad_indices"], self.ptr["peaks"],
                                        self.ptr["basins"], ctypes.byref(sizes), ctypes.c_void_p(stream.cuda_stream))
        self.ctx.check(rc, "extract")
        assert sizes.ridges == self.ref.ridges.numel() and sizes.valleys == self.ref.valleys.numel()

    def fetch_start(self, stream):
        self.ctx.check(self.lib.dmsc_b200_fetch_start(self.ctx.h, ctypes.byref(self.outputs),
                                                      ctypes.c_void_p(stream.cuda_stream)), "fetch_start")

    def fetch_finish(self, stream):
        return self.lib.dmsc_b200_fetch_finish(self.ctx.h, ctypes.c_void_p(stream.cuda_stream))

    def differing(self):
        torch.cuda.synchronize()
        return [f for f, t in self.out.items() if not torch.equal(t, getattr(self.ref, f))]


def test_two_phases_on_two_streams():
    """fetch reads what the expansion at the end of extract is still writing."""
    from dmsc_b200 import compute_dmsc
    from dmsc_b200.synthetic import field_4096_bumps

    img = field_4096_bumps(seed=6)[:1500, :1700].contiguous().cuda()
    raw = _Raw(img, 0.25, compute_dmsc(img, 0.25))
    s1, s2 = torch.cuda.Stream(), torch.cuda.Stream()
    for _ in range(3):
        raw.extract(s1)
        raw.fetch_start(s2)
        assert raw.fetch_finish(s2) == 0
        assert raw.differing() == []


def test_fetch_that_is_never_finished():
    from dmsc_b200 import compute_dmsc
    from dmsc_b200.synthetic import field_256_bumps

    img, y = field_256_bumps(seed=7).cuda(), _fields((130, 211), 8)
    ref_y = compute_dmsc(y, 0.02)
    raw = _Raw(img, 0.1, compute_dmsc(img, 0.1))
    s1, s2 = torch.cuda.Stream(), torch.cuda.Stream()
    raw.extract(s1)
    with torch.cuda.stream(s1):
        torch.cuda._sleep(DELAY)
    raw.fetch_start(s1)
    with torch.cuda.stream(s2):
        c = compute_dmsc(y, 0.02)
    assert raw.differing() == [] and diff_fields(c, ref_y) == []
    assert raw.fetch_finish(s1) == 1  # no fetch is pending
