"""tcgen05/TMEM GEMM against torch.matmul in fp32 for every operand layout and epilogue."""

import pytest
import torch

from templar_b200.ops import functional as OF

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.fixture(params=["tcgen05", "tcgen05_2sm"], autouse=True)
def backend(request):
    """Every test runs on the one-CTA-per-tile kernel and on the CTA-pair (cta_group::2) kernel."""
    prev = OF.gemm_backend()
    OF.set_gemm_backend(request.param)
    yield request.param
    OF.set_gemm_backend(prev)


def _check(M, N, K, a_mn, b_mn, epi):
    torch.manual_seed(M + N + K)
    A = torch.randn((K, M) if a_mn else (M, K), device=DEV).to(torch.bfloat16)
    B = torch.randn((K, N) if b_mn else (N, K), device=DEV).to(torch.bfloat16)
    Af = (A.t() if a_mn else A).float()
    Bf = (B if b_mn else B.t()).float()
    ref = Af @ Bf
    OF.status_word(DEV).zero_()
    if epi == "bf16":
        out = OF.gemm(A, B, a_mn=a_mn, b_mn=b_mn)
        tol = 2e-2 * (K ** 0.5)
    elif epi == "f32":
        out = OF.gemm(A, B, a_mn=a_mn, b_mn=b_mn, out_dtype=torch.float32)
        tol = 1e-3 * (K ** 0.5)
    else:
        base = torch.randn(M, N, device=DEV)
        out = OF.gemm(A, B, a_mn=a_mn, b_mn=b_mn, out=base.clone(), accumulate=True)
        ref = ref + base
        tol = 1e-3 * (K ** 0.5)
    torch.cuda.synchronize()
    assert int(OF.status_word(DEV).item()) == 0, "bounded wait expired inside the GEMM kernel"
    err = (out.float() - ref).abs().max().item()
    assert err < tol, (M, N, K, a_mn, b_mn, epi, err)


@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, True), (True, False)])
@pytest.mark.parametrize("epi", ["bf16", "f32", "acc"])
def test_gemm_layouts(a_mn, b_mn, epi):
    _check(256, 512, 320, a_mn, b_mn, epi)


@pytest.mark.parametrize("M,N,K", [(128, 256, 64), (384, 256, 2048), (2048, 2048, 2048), (1000, 776, 136),
                                   (4096, 32000, 512), (130, 264, 72), (8, 8, 8), (257, 513, 4104)])
def test_gemm_shapes(M, N, K):
    _check(M, N, K, False, False, "bf16")


# (tokens, out features, in features) of the projections of the 1B benchmark model (16384 tokens per micro-batch)
# and of the 18B tensor-parallel configuration (2048 tokens, features divided over 8 ranks where the plan shards them)
MODEL_SHAPES = [(16384, 6144, 2048), (16384, 2048, 2048), (16384, 16384, 2048), (16384, 2048, 8192), (16384, 32000, 2048),
                (2048, 1280, 8192), (2048, 8192, 1024), (2048, 7168, 8192), (2048, 8192, 3584), (2048, 16032, 8192)]


@pytest.mark.parametrize("T,N,K", MODEL_SHAPES)
def test_gemm_model_shapes_forward_dgrad_wgrad(T, N, K, backend):
    """Forward (x W^T), input gradient (dy W) and weight gradient (dy^T x, fp32 accumulate) of one projection."""
    if backend != "tcgen05_2sm" and T * N > 2 ** 27:
        pytest.skip("the one-CTA kernel is the secondary backend: large cases run on the CTA-pair kernel only")
    torch.manual_seed(T + N + K)
    x = (torch.randn(T, K, device=DEV) * 0.5).to(torch.bfloat16)
    w = (torch.randn(N, K, device=DEV) * 0.05).to(torch.bfloat16)
    OF.status_word(DEV).zero_()
    y = OF.gemm(x, w)
    ref = x.float() @ w.float().t()
    assert (y.float() - ref).abs().max().item() < 2e-2 * max(ref.abs().max().item(), 1.0)
    dy = (torch.randn(T, N, device=DEV) * 0.1).to(torch.bfloat16)
    dx = OF.gemm(dy, w, b_mn=True)
    ref = dy.float() @ w.float()
    assert (dx.float() - ref).abs().max().item() < 2e-2 * max(ref.abs().max().item(), 1.0)
    del ref
    acc = torch.ones(N, K, device=DEV)
    OF.gemm(dy, x, a_mn=True, b_mn=True, out=acc, accumulate=True)
    ref = dy.float().t() @ x.float() + 1.0
    assert (acc - ref).abs().max().item() < 2e-3 * max(ref.abs().max().item(), 1.0)
    torch.cuda.synchronize()
    assert int(OF.status_word(DEV).item()) == 0


def test_library_fallback_is_counted_and_said(backend):
    """Operands that the own kernels cannot take (a row stride that is not a multiple of 8 elements) go to the
    library with a warning and a counter; under TPLR_STRICT_NATIVE=1 they are an error."""
    import os
    import warnings

    a = torch.randn(64, 36, device=DEV).to(torch.bfloat16)[:, :32]        # row stride 36
    b = torch.randn(48, 32, device=DEV).to(torch.bfloat16)
    before = OF.library_gemm_fallbacks
    OF._gemm_fallback_seen.clear()
    with warnings.catch_warnings(record=True) as seen:
        warnings.simplefilter("always")
        c = OF.gemm(a, b)
    assert OF.library_gemm_fallbacks == before + 1 and any("own tcgen05 kernels" in str(w.message) for w in seen)
    assert (c.float() - a.float() @ b.float().t()).abs().max().item() < 0.5
    os.environ["TPLR_STRICT_NATIVE"] = "1"
    try:
        with pytest.raises(RuntimeError):
            OF.gemm(a, b)
    finally:
        del os.environ["TPLR_STRICT_NATIVE"]


def test_linear_backward_matches_autograd():
    x = torch.randn(3, 100, 256, device=DEV, dtype=torch.bfloat16, requires_grad=True)
    w = (torch.randn(512, 256, device=DEV) * 0.05).to(torch.bfloat16).requires_grad_()
    y = OF.linear(x, w)
    dy = torch.randn_like(y)
    y.backward(dy)
    xf, wf = x.detach().float().requires_grad_(), w.detach().float().requires_grad_()
    (xf @ wf.t()).backward(dy.float())
    assert torch.allclose(x.grad.float(), xf.grad, atol=0.1, rtol=3e-2)
    assert torch.allclose(w.grad.float(), wf.grad, atol=0.5, rtol=3e-2)


def test_gemm_from_a_fresh_thread():
    """The tensor-map encode is a driver call; a thread that has not touched CUDA yet (like an
    autograd worker) must still be able to launch the GEMM."""
    import threading

    A = torch.randn(256, 128, device=DEV).to(torch.bfloat16)
    B = torch.randn(512, 128, device=DEV).to(torch.bfloat16)
    box = {}

    def work():
        try:
            box["out"] = OF.gemm(A, B)
        except Exception as e:  # noqa: BLE001
            box["err"] = e

    t = threading.Thread(target=work)
    t.start()
    t.join()
    torch.cuda.synchronize()
    assert "err" not in box, box.get("err")
    assert (box["out"].float() - A.float() @ B.float().t()).abs().max().item() < 0.5


@pytest.mark.parametrize("M,F,K", [(512, 256, 512), (300, 384, 192), (16384, 8192, 2048), (1000, 128, 64)])
def test_fused_swiglu_projection_matches_fp32_reference(M, F, K, backend):
    """[w1; w3] projection with silu(g) * u in the GEMM epilogue: both outputs against PyTorch in fp32, and the
    gradients of the op against autograd through the fp32 formula.  The last tile row is ragged for M = 300 / 1000."""
    if backend != "tcgen05_2sm":
        pytest.skip("the fused epilogue is a mode of the CTA-pair kernel")
    torch.manual_seed(M + F)
    x = (torch.randn(M, K, device=DEV) * 0.5).to(torch.bfloat16).requires_grad_()
    w = (torch.randn(2 * F, K, device=DEV) / K ** 0.5).to(torch.bfloat16).requires_grad_()
    OF.status_word(DEV).zero_()
    before = OF.library_gemm_fallbacks
    from templar_b200.ops import native
    n0 = native.launch_count
    h = OF.linear_swiglu(x, w)
    assert native.launch_count - n0 == 1            # projection and activation in one launch
    dh = torch.randn_like(h)
    h.backward(dh)
    torch.cuda.synchronize()
    assert int(OF.status_word(DEV).item()) == 0 and OF.library_gemm_fallbacks == before
    xf, wf = x.detach().float().requires_grad_(), w.detach().float().requires_grad_()
    gu = xf @ wf.t()
    ref = torch.nn.functional.silu(gu[:, :F]) * gu[:, F:]
    ref.backward(dh.float())
    assert (h.float() - ref).abs().max().item() < 2e-2 * max(1.0, ref.abs().max().item())
    # the two-launch path computes the activation from bf16-rounded g and u: the fused result is at least as close
    two = OF.swiglu(OF.linear(x.detach(), w.detach())).float()
    assert (h.float() - ref).abs().mean().item() <= 1.05 * (two - ref).abs().mean().item() + 1e-6
    for got, want in ((x.grad, xf.grad), (w.grad, wf.grad)):
        rel = (got.float() - want).norm() / want.norm()
        assert rel.item() < 2e-2, rel.item()


@pytest.mark.parametrize("T,D,F", [(512, 256, 256), (300, 192, 384), (16384, 2048, 8192), (1000, 64, 128)])
def test_feed_forward_with_both_swiglu_epilogues_matches_fp32_reference(T, D, F, backend):
    """swiglu(x W13^T) W2^T as one node: activation in the first projection's epilogue, its backward in the epilogue of
    the second projection's data gradient.  Output and all three gradients against autograd through the fp32 formula,
    and against the node-per-op path (which other tests pin to fp32 PyTorch)."""
    if backend != "tcgen05_2sm":
        pytest.skip("the fused epilogues are modes of the CTA-pair kernel")
    from templar_b200.ops import native

    torch.manual_seed(T + F)
    x = (torch.randn(T, D, device=DEV) * 0.5).to(torch.bfloat16)
    w13 = (torch.randn(2 * F, D, device=DEV) / D ** 0.5).to(torch.bfloat16)
    w2 = (torch.randn(D, F, device=DEV) / F ** 0.5).to(torch.bfloat16)
    dy = torch.randn(T, D, device=DEV).to(torch.bfloat16)
    OF.status_word(DEV).zero_()

    def run(fused):
        prev = OF.FUSED_PROJECTIONS
        OF.FUSED_PROJECTIONS = fused
        try:
            xs, a, b = (t.clone().requires_grad_() for t in (x, w13, w2))
            n0 = native.launch_count
            y = OF.feed_forward(xs, a, b)
            fwd = native.launch_count - n0
            y.backward(dy)
            return y.float(), xs.grad.float(), a.grad.float(), b.grad.float(), fwd, native.launch_count - n0
        finally:
            OF.FUSED_PROJECTIONS = prev

    yf, *gf, fwd_f, all_f = run(True)
    ys, *gs, fwd_s, all_s = run(False)
    torch.cuda.synchronize()
    assert int(OF.status_word(DEV).item()) == 0
    assert fwd_f == 2 and all_f == 6 and fwd_s == 3 and all_s == 8      # one launch less in each direction
    xf, af, bf = (t.float().requires_grad_() for t in (x, w13, w2))
    gu = xf @ af.t()
    ref = (torch.nn.functional.silu(gu[:, :F]) * gu[:, F:]) @ bf.t()
    ref.backward(dy.float())
    rel = lambda a_, b_: ((a_ - b_).norm() / b_.norm()).item()      # noqa: E731
    errs_f = [rel(yf, ref)] + [rel(g, r.grad) for g, r in zip(gf, (xf, af, bf))]
    errs_s = [rel(ys, ref)] + [rel(g, r.grad) for g, r in zip(gs, (xf, af, bf))]
    assert max(errs_f) < 2e-2, (errs_f, errs_s)
    assert all(a_ < 1.3 * b_ + 1e-3 for a_, b_ in zip(errs_f, errs_s)), (errs_f, errs_s)


@pytest.mark.parametrize("M,N,K", [(768, 768, 8192), (264, 520, 4104), (256, 256, 576), (2304, 768, 520)])
def test_accumulating_gemm_with_k_splits(M, N, K, backend):
    """Weight-gradient products with few tiles (several work units add into one tile), ragged tiles and a ragged last split."""
    _check(M, N, K, True, True, "acc")


@pytest.mark.parametrize("T,D,F", [(300, 192, 384), (1000, 64, 128)])
def test_feed_forward_without_grad_gives_the_same_output(T, D, F, backend):
    """Without a backward pass the packed projection is not stored; the activation and the output are the same bits."""
    if backend != "tcgen05_2sm":
        pytest.skip("the fused epilogue is a mode of the CTA-pair kernel")
    torch.manual_seed(T)
    x, w13, w2 = (torch.randn(*s, device=DEV).to(torch.bfloat16).requires_grad_() for s in ((T, D), (2 * F, D), (D, F)))
    want = OF.feed_forward(x, w13, w2).detach()
    with torch.no_grad():
        assert torch.equal(OF.feed_forward(x, w13, w2), want)
    assert int(OF.status_word(DEV).item()) == 0


@pytest.mark.parametrize("M,N,K,b_mn", [(256, 256, 4096, False), (777, 264, 6152, True), (8, 8, 8192, False), (300, 1024, 5000, True)])
def test_bf16_gemm_through_split_workspace(M, N, K, b_mn, backend):
    """Few tiles and a long K: partial products summed in fp32 and rounded once; ragged tiles, a ragged last split, a
    result that is a view with a leading dimension of its own, and the same bits on a second run."""
    from templar_b200.ops import native

    if backend == "tcgen05_2sm":
        assert native.lib().tplr_gemm2_out_splits(M, N, K) > 1
    _check(M, N, K, False, b_mn, "bf16")
    A = (torch.randn(M, K, device=DEV) / K ** 0.5).to(torch.bfloat16)
    B = torch.randn((K, N) if b_mn else (N, K), device=DEV).to(torch.bfloat16)
    wide = torch.full((M, N + 16), 7.0, device=DEV, dtype=torch.bfloat16)
    OF.gemm(A, B, b_mn=b_mn, out=wide[:, 8:-8])
    ref = A.float() @ (B if b_mn else B.t()).float()
    assert torch.allclose(wide[:, 8:-8].float(), ref, rtol=2 ** -8, atol=1e-3)        # one rounding; fp32 sums of K products
    assert (wide[:, :8] == 7).all() and (wide[:, -8:] == 7).all()
    assert torch.equal(OF.gemm(A, B, b_mn=b_mn), wide[:, 8:-8])


@pytest.mark.parametrize("M,N,K", [(768, 768, 8192), (264, 520, 4104), (2304, 768, 8192), (1536, 4096, 4096)])
def test_accumulating_gemm_repeats_its_bits(M, N, K, backend):
    """A weight gradient added into a buffer that holds an earlier one: the parts of K are added in order, not as they arrive."""
    if backend != "tcgen05_2sm":
        pytest.skip("only the CTA-pair kernel cuts K")
    torch.manual_seed(M + N)
    A, B = (torch.randn(K, n, device=DEV).to(torch.bfloat16) for n in (M, N))
    before = torch.randn(M, N, device=DEV)
    first = OF.gemm(A, B, a_mn=True, b_mn=True, out=before.clone(), accumulate=True)
    for _ in range(30):
        assert torch.equal(OF.gemm(A, B, a_mn=True, b_mn=True, out=before.clone(), accumulate=True), first)


@pytest.mark.parametrize("grad", [True, False])
def test_feed_forward_refuses_weights_of_other_widths(grad, backend):
    """The fused projection takes its inner dimension from the input: a weight of another one would be read out of range."""
    bf = lambda *shape: torch.zeros(*shape, device=DEV, dtype=torch.bfloat16)      # noqa: E731
    x, w13, w2 = bf(64, 256), bf(512, 256), bf(256, 256)
    with torch.set_grad_enabled(grad):
        for a, b in ((bf(512, 248), w2), (bf(512, 264), w2), (w13, bf(256, 264)), (w13, bf(256, 248))):
            with pytest.raises(ValueError):
                OF.feed_forward(x, a, b)


@pytest.mark.parametrize("b_mn", [False, True])
@pytest.mark.parametrize("M,N,K,epi", [(1111, 1536, 1536, "bf16"), (300, 760, 200, "bf16"), (300, 1160, 72, "bf16"),     # 128 wide, remainders
                                       (2100, 3656, 776, "bf16"), (8192, 776, 768, "bf16"), (300, 5640, 64, "bf16"),     # 192 wide (K-major)
                                       (520, 1032, 136, "f32"), (2304, 776, 2000, "acc"), (520, 136, 4104, "acc"),       # fp32 tiles, parts of K
                                       (260, 1160, 8200, "bf16")])
def test_narrow_tiles(M, N, K, epi, b_mn):
    """Products whose 256-wide tiles would leave SMs idle: last tiles of 8 to 184 columns, with and without parts of K."""
    _check(M, N, K, epi == "acc", b_mn, epi)


def test_chain_of_dependent_launches(backend):
    """Kernels that may start while the one before them runs: a chain in which each reads what the one before wrote (products, parts
    of K added by a second kernel, attention both ways, a torch kernel between), against the same chain with a wait behind every call."""
    torch.manual_seed(0)
    bf = lambda *s, std=1.0: (torch.randn(*s, device=DEV) * std).to(torch.bfloat16)      # noqa: E731
    x, w, up, wide = bf(512, 384), bf(384, 384, std=0.05), bf(8192, 384, std=0.05), bf(384, 8192, std=0.01)
    mg = torch.zeros(384, 384, device=DEV)

    def chain(wait):
        h, grad = x, mg.clone()
        for _ in range(4):
            h = OF.gemm(h, w)
            wait()
            h = OF.gemm(OF.gemm(h, up), wide)                  # K = 8192: parts
            wait()
            q = OF.attention_packed(OF.gemm(h, w).view(2, 256, 384), 2, 2, 64)
            wait()
            h = OF.gemm(torch.cat([q.reshape(512, 128)] * 3, dim=1), w) + x
            wait()
            OF.gemm(h, h, a_mn=True, b_mn=True, out=grad, accumulate=True)
            wait()
        return h, grad

    want = chain(torch.cuda.synchronize)
    for _ in range(20):
        assert all(torch.equal(a, b) for a, b in zip(chain(lambda: None), want))
    assert int(OF.status_word(DEV).item()) == 0
