"""Kernels that may start while the one before them runs: whole blocks forward and backward, in which each kernel reads what the one
before wrote, give the bits of the same chain with a wait behind every entry of the library."""

import pytest
import torch

from templar_b200.ops import functional as OF
from templar_b200.ops import native

pytestmark = pytest.mark.gpu
DEV = "cuda"


class _Waiting:
    """The library, with a wait behind every call."""

    def __init__(self, lib):
        self._lib = lib

    def __getattr__(self, name):
        fn = getattr(self._lib, name)

        def call(*args):
            rc = fn(*args)
            torch.cuda.synchronize()
            return rc

        return call


@pytest.mark.parametrize("H,KV,hd", [(8, 8, 64), (8, 2, 64), (4, 4, 128), (4, 1, 128)])
def test_blocks_forward_and_backward(H, KV, hd, monkeypatch):
    """Rotary, SwiGLU and delta epilogues, attention both ways with whole and with cut groups of query heads, weight gradients, an
    accumulating product whose parts of K a second kernel adds.  Sequences of two key blocks: dQ is a sum of two terms, whose
    order does not matter, and all other sums have an order, so the bits are the same."""
    torch.manual_seed(H * hd + KV)
    B, S, D, F, L = 2, 256, 512, 1024, 3
    bf = lambda *s, std=1.0: (torch.randn(*s, device=DEV) * std).to(torch.bfloat16)      # noqa: E731
    cos, sin = OF.rope_tables(S, hd, 10000.0, DEV)
    cos, sin = cos.contiguous(), sin.contiguous()
    x0, dy = bf(B, S, D), bf(B, S, D)
    weights = [[bf((H + 2 * KV) * hd, D, std=D ** -0.5), bf(D, H * hd, std=(H * hd) ** -0.5), bf(2 * F, D, std=D ** -0.5),
                bf(D, F, std=F ** -0.5)] for _ in range(L)]
    up = bf(16 * D, D, std=D ** -0.5)
    lib = native.lib()
    assert lib.tplr_gemm2_acc_splits(D, D, 16 * D) > 1
    assert (lib.tplr_attention_bwd_scratch_cols(B, S, H, KV, hd) > H * hd) == (KV < H)

    def chain():
        x = x0.clone().requires_grad_()
        layers = [[w.clone().requires_grad_() for w in ws] for ws in weights]
        for ws in layers:
            for w in ws:
                w.main_grad = torch.zeros(w.shape, device=DEV)
        h = x
        for wqkv, wo, w13, w2 in layers:
            h = OF.attention_block(h, wqkv, wo, cos, sin, H, KV, hd)
            h = OF.feed_forward(h, w13, w2)
        h.backward(dy)
        long = OF.gemm(up, x.grad.view(-1, D), b_mn=True)                   # [16 D, D], read by the next kernel
        total = OF.gemm(long, long, a_mn=True, b_mn=True, out=torch.ones(D, D, device=DEV), accumulate=True)
        return [h.detach(), x.grad, long, total, *(w.main_grad for ws in layers for w in ws)]

    with monkeypatch.context() as m:
        m.setattr(native, "host", lambda: None)                             # the nodes in Python call the entries one by one
        m.setattr(native, "lib", lambda: _Waiting(lib))
        want = chain()
    torch.cuda.synchronize()
    assert all(torch.isfinite(t).all() and t.float().abs().max() > 0 for t in want)
    # an entry of two kernels has no wait between them: its result on its own
    ref = want[2].double().t() @ want[2].double() + 1
    assert ((want[3].double() - ref).norm() / ref.norm()).item() < 16 * D / 16 * 2 ** -23      # fp32 sums, 16 products at a time
    for _ in range(10):
        for got, w in zip(chain(), want):
            assert torch.equal(got, w)
    assert int(OF.status_word(DEV).item()) == 0
