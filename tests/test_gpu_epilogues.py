"""The fused epilogues of the CTA-pair GEMM at every tile width that the rule picks for their layouts (256, 192 and 128 columns),
with ragged last tiles in both directions, against the same formula in 64 bits.  Short K: the widths depend on rows and columns."""

import pytest
import torch

from templar_b200.ops import functional as OF
from templar_b200.ops import native

pytestmark = pytest.mark.gpu
DEV = "cuda"
K = 72
# An output is rounded to bf16 once, from fp32 sums of K products of values around 1 (each off by less than K * 2^-24 * sum |a b|,
# about 3e-5) and, in the activations, from an approximate exponential of comparable error, multiplied by values up to 5.
ROUNDING, SUMS = 2 ** -8, 3e-4


def bf(*shape, std=1.0):
    return (torch.randn(*shape, device=DEV) * std).to(torch.bfloat16)


def close(got, want, atol=SUMS):
    err = (got.double() - want).abs() - want.abs() * ROUNDING
    assert err.max().item() <= atol, err.max().item()


def call(entry, *args):
    st = OF.status_word(DEV)
    st.zero_()
    native.check(getattr(native.lib(), entry)(*(a.data_ptr() if torch.is_tensor(a) else a for a in args), st.data_ptr(),
                                              native.stream_ptr()), entry)
    assert int(st.item()) == 0


@pytest.mark.parametrize("B,S,H,KV,hd", [(3, 100, 9, 3, 64), (2, 1500, 9, 3, 64), (3, 1400, 9, 3, 64),       # 128, 192 and 256 columns, 960 in all
                                         (3, 700, 17, 1, 64), (3, 1000, 17, 1, 64),                          # 192 and 256, 1216 in all
                                         (1, 300, 7, 1, 128), (3, 700, 7, 1, 128), (1, 257, 4, 2, 128)])     # 128 and 256, 1152 and 1024
def test_rotary_epilogue(B, S, H, KV, hd):
    torch.manual_seed(S)
    T, C, rot = B * S, (H + 2 * KV) * hd, (H + KV) * hd
    x, w = bf(T, K), bf(C, K, std=K ** -0.5)
    cos, sin = OF.rope_tables(S, hd, 10000.0, DEV)
    cos, sin = cos.contiguous(), sin.contiguous()
    wide = torch.full((T, C + 8), 7.0, device=DEV, dtype=torch.bfloat16)
    call("tplr_gemm2_rope", x, w, wide, T, C, K, K, K, C + 8, cos, sin, S, rot, hd)
    want = (x.double() @ w.double().t()).view(B, S, C)
    pairs = want[..., :rot].reshape(B, S, -1, hd // 2, 2)
    c, s = (t[:S].double().view(1, S, 1, hd // 2) for t in (cos, sin))
    a, b = pairs.unbind(-1)
    turned = torch.stack((a * c - b * s, a * s + b * c), dim=-1).reshape(B, S, rot)
    close(wide[:, :C].view(B, S, C), torch.cat((turned, want[..., rot:]), dim=-1))
    assert (wide[:, C:] == 7).all()


@pytest.mark.parametrize("T,H,hd", [(300, 9, 64), (1500, 17, 64), (4200, 9, 64), (2100, 17, 64),       # 128 and 256 columns, 576 and 1088 in all
                                    (300, 7, 128), (2100, 13, 128), (6099, 7, 128)])                   # 128 and 256, 896 and 1664
def test_delta_epilogue(T, H, hd):
    torch.manual_seed(T)
    S, N = T // 3, H * hd
    dy, wo, o = bf(T, K), bf(K, N, std=K ** -0.5), bf(T, N)
    wide = torch.full((T, N + 8), 7.0, device=DEV, dtype=torch.bfloat16)
    delta = torch.empty(3, H, S, device=DEV)
    call("tplr_gemm2_attn_dout", dy, wo, o, wide, delta, T, N, K, S, hd, K, N, N, N + 8)
    do = wide[:, :N]
    close(do, dy.double() @ wo.double())
    assert (wide[:, N:] == 7).all()
    terms = (do.double() * o.double()).view(3, S, H, hd).transpose(1, 2)             # of the values as stored
    assert ((delta.double() - terms.sum(-1)).abs() <= hd * 2 ** -24 * terms.abs().sum(-1)).all()


@pytest.mark.parametrize("T,F", [(300, 384), (4200, 384), (2100, 1152), (1000, 2176), (300, 2944)])       # features by 64, then by 128
@pytest.mark.parametrize("stored", [True, False])
def test_swiglu_epilogue(T, F, stored):
    torch.manual_seed(T)
    x, w = bf(T, K), bf(2 * F, K, std=K ** -0.5)
    gu = torch.full((T, 2 * F + 8), 7.0, device=DEV, dtype=torch.bfloat16)
    h = torch.full((T, F + 8), 7.0, device=DEV, dtype=torch.bfloat16)
    call("tplr_gemm2_swiglu", x, w, gu if stored else None, h, T, F, K, K, K, 2 * F + 8, F + 8)
    want = x.double() @ w.double().t()
    close(h[:, :F], torch.nn.functional.silu(want[:, :F]) * want[:, F:])
    if stored:
        close(gu[:, :2 * F], want)
    assert (gu[:, 2 * F:] == 7).all() and (h[:, F:] == 7).all() and (stored or (gu == 7).all())


@pytest.mark.parametrize("T,F", [(300, 640), (1000, 448), (4200, 640), (2100, 1152), (2100, 1216), (1000, 2944)])      # 128 and 256 columns
def test_swiglu_backward_epilogue(T, F):
    torch.manual_seed(T)
    dy, w2, gu = bf(T, K), bf(K, F, std=K ** -0.5), bf(T, 2 * F)
    dgu = torch.full((T, 2 * F + 8), 7.0, device=DEV, dtype=torch.bfloat16)
    call("tplr_gemm2_swiglu_bwd", dy, w2, gu, dgu, T, F, K, K, F, 2 * F, 2 * F + 8)
    g, u = gu.double().split(F, dim=1)
    dh, sg = dy.double() @ w2.double(), torch.sigmoid(g)
    close(dgu[:, :F], dh * u * (sg + g * sg * (1 - sg)))
    close(dgu[:, F:2 * F], dh * g * sg)
    assert (dgu[:, 2 * F:] == 7).all()
