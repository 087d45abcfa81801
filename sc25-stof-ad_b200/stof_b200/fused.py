"""Fused GEMM / LayerNorm operators (host side of `stof_gemm_bias_act` and
`stof_bias_residual_layernorm`; argument checks and launches are in `csrc/host/stof_native.cpp`)."""
from __future__ import annotations

import torch

from . import _lib


EPILOGUES = {"gelu_erf": _lib.EPI_BIAS_GELU_ERF, "erf": _lib.EPI_BIAS_GELU_ERF, "gelu_tanh": _lib.EPI_BIAS_GELU_TANH,
             "tanh": _lib.EPI_BIAS_GELU_TANH, "relu": _lib.EPI_BIAS_RELU, "none": _lib.EPI_BIAS}


def gemm_bias(a, w, bias=None, out=None):
    """a (..., K) @ w (K, N) + bias (N) -> (..., N) fp16 (fp32 accumulation)."""
    return (_lib._native or _lib.native()).gemm(a, w, bias, _lib.EPI_BIAS, None, out)


def gemm_bias_gelu(a, w, bias=None, mode: str = "erf", out=None):
    """GEMM + bias + GELU in one kernel; mode "erf" (F.gelu, src/benchmk_end2end.py:81) or
    "tanh" (src/triton_template/gemm_gemm.py:146-150)."""
    if mode not in ("erf", "tanh"):
        raise _lib.StofError(f"gemm_bias_gelu: unknown mode {mode!r}")
    return (_lib._native or _lib.native()).gemm(a, w, bias, _lib.EPI_BIAS_GELU_ERF if mode == "erf" else _lib.EPI_BIAS_GELU_TANH, None, out)


def gemm_bias_relu(a, w, bias=None, out=None):
    """GEMM + bias + ReLU in one kernel (the FFN activation of the T5 loops, src/benchmk_end2end.py:203,313)."""
    return (_lib._native or _lib.native()).gemm(a, w, bias, _lib.EPI_BIAS_RELU, None, out)


def gemm_bias_act(a, w, bias=None, activation: str = "gelu_erf", out=None):
    """GEMM + bias + activation by name: "gelu_erf" (BERT), "gelu_tanh" (GPT-2 `new_gelu`), "relu" (T5), "none"."""
    epi = EPILOGUES.get(activation)
    if epi is None:
        raise _lib.StofError(f"gemm_bias_act: unknown activation {activation!r}")
    return (_lib._native or _lib.native()).gemm(a, w, bias, epi, None, out)


def gemm_bias_residual(a, w, bias, residual, out=None):
    """GEMM + bias + residual add in one kernel."""
    if residual is None:
        raise _lib.StofError("gemm: the residual epilogue needs a residual")
    return (_lib._native or _lib.native()).gemm(a, w, bias, _lib.EPI_BIAS_RESIDUAL, residual, out)


def bias_residual_layernorm(x, bias=None, residual=None, gamma=None, beta=None, eps: float = 1e-5, out=None):
    """y = LayerNorm(x + bias + residual) * gamma + beta over the last dimension, one pass over HBM."""
    return (_lib._native or _lib.native()).layernorm(x, bias, residual, gamma, beta, eps, out)


def gemm_bias_residual_layernorm(a, w, bias, residual, gamma, beta, eps: float, out=None):
    """LayerNorm(a @ w + bias + residual) * gamma + beta (src/benchmk_end2end.py:73-76, 83-86; the statistics inside the GEMM
    kernel as in src/triton_template/gemm_add_layernorm.py:77-123): for N a multiple of 256 up to 1024 and K <= 2048 ONE tcgen05
    kernel whose epilogue takes the row statistics across a cluster of thread blocks (`stof_gemm_bias_residual_layernorm`); other
    N, and longer K where that is faster, run the GEMM with the bias + residual epilogue and the LayerNorm kernel in place.
    bias, residual, gamma, beta may be None."""
    return (_lib._native or _lib.native()).gemm_ln(a, w, bias, residual, gamma, beta, eps, out)


def gemm_bias_residual_then_layernorm(a, w, bias, residual, gamma, beta, eps: float, out=None):
    """The same result from two kernels: tcgen05 GEMM with the bias + residual epilogue (fp16 out), then the one-pass LayerNorm
    kernel in place.  Kept for comparison with the fused form (it rounds the GEMM output to fp16 before the statistics)."""
    x = gemm_bias_residual(a, w, bias, residual, out=out) if residual is not None else gemm_bias(a, w, bias, out=out)
    return bias_residual_layernorm(x, None, None, gamma, beta, eps, out=x)


# ------------------------------------------------------------------------------------------
# Operators with the signatures of the reference's Triton templates
# ------------------------------------------------------------------------------------------
def matmul_bias_layernorm(A, B, bias, eps: float = 1e-5):
    """`triton_matmul_bias_layernorm(A, B, bias, eps)` (src/triton_template/gemm_add_layernorm.py:126-144):
    C[b] = normalise_rows(A[b] @ B[b] + bias[:N]), no gamma/beta.  A (batch,M,K), B (batch,K,N);
    a batch-expanded weight (stride 0) runs as one GEMM over batch*M rows."""
    batch, M, K = A.shape
    _, Kb, N = B.shape
    if K != Kb:
        raise _lib.StofError(f"matmul_bias_layernorm: K mismatch ({K} vs {Kb})")
    bvec = bias.reshape(-1)[:N].contiguous()
    C = torch.empty(batch, M, N, dtype=A.dtype, device=A.device)
    if B.stride(0) == 0 or batch == 1:
        gemm_bias_residual_layernorm(A, B[0], bvec, None, None, None, eps, out=C)
    else:
        for b in range(batch):
            gemm_bias_residual_layernorm(A[b], B[b], bvec, None, None, None, eps, out=C[b])
    return C


def matmul_gelu_matmul(a, b, d, bias):
    """`triton_matmul_batch(a, b, d, bias)` (src/triton_template/gemm_gemm.py:158-174):
    gelu_tanh(a @ b + bias[:N]) @ d with the intermediate rounded to fp16.  a (batch,M,K), b (K,N), d (N,H).
    Two back-to-back tcgen05 GEMMs; the (batch*M, N) intermediate stays in L2 for typical FFN sizes."""
    N = b.shape[-1]
    t = gemm_bias_gelu(a, b, bias.reshape(-1)[:N].contiguous(), mode="tanh")
    return gemm_bias(t, d, None)


def batched_bias_layernorm(x, bias, weight, bias_ln, eps: float = 1e-5):
    """`triton_batched_bias_layernorm(x, bias, weight, bias_ln, eps)`
    (src/triton_template/add_layernorm.py:86-107): LN(x + bias) * weight + bias_ln."""
    return bias_residual_layernorm(x, bias, None, weight, bias_ln, eps)
