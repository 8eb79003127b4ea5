"""Newton–Schulz orthogonalisation for Muon on the tcgen05 GEMM.

Five quintic iterations with per-iteration coefficients (the schedule of the reference's
src/tplr/muon/newton_schulz_triton.py:336-374):

    A = X X^T                    "line 1"  -> ``gemm(X, X)``          (both operands K-major: one tensor, two roles)
    B = b A + c A A              "line 2"  -> ``gemm(A, A)`` + axpby  (A is symmetric, so A A = A A^T)
    X = a X + B X                "line 3"  -> ``gemm(B, X, b_mn=True)`` + axpby

bf16 operands, fp32 accumulation in TMEM.  The reference runs lines 1-2 as Triton kernels that compute one triangle
of the symmetric results and mirror it on the store, and line 3 through cuBLAS; here all three are the same
hand-written tcgen05 kernel, lines 1-2 in its one-triangle mode (``_ns_2d_symmetric``), and no transposed copy is
made.  ``python -m templar_b200.muon.bench`` times the variants and the reference's kernels.
Batched inputs (leading dimensions) are processed matrix by matrix.
"""

from __future__ import annotations

import torch

from ..ops import functional as OF

NS_CONSTS = [(4.0848, -6.8946, 2.9270), (3.9505, -6.3029, 2.6377), (3.7418, -5.5913, 2.3037),
             (2.8769, -3.1427, 1.2046), (2.8366, -3.0525, 1.2012)]


def _one_triangle_ok(G: torch.Tensor) -> bool:
    return (G.is_cuda and OF.gemm_backend() == "tcgen05_2sm" and min(G.shape) >= 512 and G.shape[0] % 8 == 0
            and G.shape[1] % 8 == 0 and SYMMETRIC_PRODUCTS)


SYMMETRIC_PRODUCTS = True        # lines 1 and 2 as one-triangle products (module switch, for the comparison benchmark)


class _SymmetricChain:
    """The five iterations for one matrix shape on static buffers, captured once in a CUDA graph and replayed:
    24 launches (per iteration: one-triangle X X^T, mirror, one-triangle A A, mirror with the line's scalars and the
    identity term, full product) with no host work between them.  Before the graph ``tplr_ns_prepare`` writes the
    scaled operand into the chain's buffer; after it the last product writes the caller's new tensor, so nothing is
    copied in or out.

    Lines 1 and 2 compute only the 256 x 256 tiles on or above the diagonal of their symmetric results
    (``tplr_gemm2_syrk``: half the tensor-core work) and ``tplr_sym_axpby`` mirrors the triangle while it applies
    the line's scalars.  Where those tiles are too few for the chip, K is cut in two and the triangle accumulates in fp32
    (``tplr_gemm2_syrk_acc``; ``tplr_sym_axpby_acc`` leaves it zeroed for the next product); the result is the same bits on
    every call and rank, which replicas that orthogonalise for themselves rely on.  Line 3, ``a X + B X``, is
    one product ``(B + a I) X``: the mirror kernel of line 2 adds ``a`` on the diagonal, so no element-wise pass over X
    remains."""

    def __init__(self, M: int, K: int, device):
        from ..ops import native

        self.M, self.K, self.native = M, K, native
        z = lambda *shape: torch.empty(*shape, dtype=torch.bfloat16, device=device)       # noqa: E731
        self.x = [z(M, K), z(M, K)]
        self.U, self.A, self.B = z(M, M), z(M, M), z(M, M)
        self.split = {k: native.lib().tplr_gemm2_syrk_splits(M, k) > 1 for k in (M, K)}
        self.acc = torch.zeros(M, M, dtype=torch.float32, device=device) if any(self.split.values()) else None
        self.scratch = torch.empty(native.lib().tplr_sumsq_blocks(), dtype=torch.float32, device=device)
        self.status = OF.status_word(device)
        self.graph = None
        self._run()                                    # warm-up outside the capture (first-use set-up of the kernels)
        torch.cuda.synchronize(device)
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            self._run()
        self.graph = g

    def _run(self) -> None:
        native, L, M, K = self.native, self.native.lib(), self.M, self.K
        st = self.status.data_ptr()
        src, dst = self.x

        def product(x, k, alpha, aux, beta, diag, out):
            """out = alpha x x^T + beta aux + diag I for x [M, k]."""
            s = native.stream_ptr()
            aux = None if aux is None else aux.data_ptr()
            if self.split[k]:
                native.check(L.tplr_gemm2_syrk_acc(x.data_ptr(), self.acc.data_ptr(), M, k, k, M, st, s), "syrk_acc")
                native.check(L.tplr_sym_axpby_acc(self.acc.data_ptr(), M, alpha, aux, beta, diag, out.data_ptr(), s), "sym_axpby_acc")
            else:
                native.check(L.tplr_gemm2_syrk(x.data_ptr(), self.U.data_ptr(), M, k, k, M, st, s), "syrk")
                native.check(L.tplr_sym_axpby(self.U.data_ptr(), M, M, alpha, aux, M, beta, diag, out.data_ptr(), M, s), "sym_axpby")

        for n, (a, b, c) in enumerate(NS_CONSTS):
            product(src, K, 1.0, None, 0.0, 0.0, self.A)
            product(self.A, M, c, self.A, b, a, self.B)                                   # A A = A A^T
            if n + 1 < len(NS_CONSTS):                                                    # the last one: __call__
                OF.gemm(self.B, src, b_mn=True, out=dst)                                  # (B + a I) X
                src, dst = dst, src
        self.last = src

    def __call__(self, G: torch.Tensor, epsilon: float) -> torch.Tensor:
        """G: contiguous bf16 or fp32; the result is [M, K] (G's transpose when G is taller than wide)."""
        rows, cols = G.shape
        self.native.check(self.native.lib().tplr_ns_prepare(
            G.data_ptr(), int(G.dtype == torch.float32), rows, cols, int(rows > cols), epsilon, self.scratch.data_ptr(),
            self.x[0].data_ptr(), self.native.stream_ptr()), "ns_prepare")
        self.graph.replay()
        return OF.gemm(self.B, self.last, b_mn=True)


_chains: dict = {}


def _ns_2d_symmetric(G: torch.Tensor, epsilon: float) -> torch.Tensor:
    M, K = min(G.shape), max(G.shape)
    key = (M, K, G.device.index, torch.cuda.current_stream(G.device).cuda_stream)
    chain = _chains.get(key)
    if chain is None:
        if len(_chains) >= 32:                          # a model has a handful of matrix shapes; bound the cache anyway
            _chains.clear()
        chain = _chains[key] = _SymmetricChain(M, K, G.device)
    X = chain(G, epsilon)
    return X.mT if G.shape[0] > G.shape[1] else X


def _ns_2d(G: torch.Tensor, epsilon: float) -> torch.Tensor:
    if _one_triangle_ok(G):
        if G.dtype not in (torch.bfloat16, torch.float32):
            G = G.to(torch.bfloat16)
        if not G.is_contiguous() or G.data_ptr() % 16:
            G = G.clone(memory_format=torch.contiguous_format)
        return _ns_2d_symmetric(G, epsilon)
    X = G.to(torch.bfloat16)
    transposed = G.size(-2) > G.size(-1)
    if transposed:
        X = X.mT
    X = (X / (X.float().norm() + epsilon).to(X.dtype)).contiguous()
    for a, b, c in NS_CONSTS:
        A = OF.gemm(X, X)                       # X X^T
        AA = OF.gemm(A, A)                      # A A^T = A A
        B = (b * A + c * AA).contiguous()
        X = (a * X + OF.gemm(B, X, b_mn=True)).contiguous()
    return X.mT if transposed else X


@torch.no_grad()
def newton_schulz(G: torch.Tensor, epsilon: float = 1e-7) -> torch.Tensor:
    """Approximate ``U V^T`` of ``G = U S V^T`` (singular values pushed towards 1)."""
    if G.ndim < 2:
        raise ValueError("newton_schulz needs a matrix")
    if G.ndim == 2:
        return _ns_2d(G, epsilon)
    flat = G.reshape(-1, G.size(-2), G.size(-1))
    return torch.stack([_ns_2d(g, epsilon) for g in flat]).reshape(G.shape)


def zeropower_via_newtonschulz5(G: torch.Tensor, steps: int = 5) -> torch.Tensor:
    """Fixed-coefficient variant ``(3.4445, -4.7750, 2.0315)`` (plain PyTorch; kept for comparison)."""
    a, b, c = 3.4445, -4.7750, 2.0315
    X = G.bfloat16() if G.is_cuda else G.float()
    t = G.size(-2) > G.size(-1)
    if t:
        X = X.mT
    X = X / (X.norm(dim=(-2, -1), keepdim=True) + 1e-7)
    for _ in range(steps):
        A = X @ X.mT
        X = a * X + (b * A + c * A @ A) @ X
    return X.mT if t else X


newton_schulz_triton = newton_schulz     # the name used by callers written against the reference
