"""Post-LN transformer forward passes built from the fused operators: the BERT encoder (reference loop:
src/benchmk_end2end.py:31-88, QKV projection as in src/model-candidate/1-BERT-large.py:17-18), its GPT-2 and T5-encoder
variants (same loop with the tanh GELU, :93-147, or ReLU, :152-208) and the T5 decoder layer (:230-316)."""
from __future__ import annotations

from dataclasses import dataclass
from typing import List

import torch

from . import _lib
from .fused import EPILOGUES
from .masks import get_sparse_storage


@dataclass
class EncoderWeights:
    """One layer: Wqkv (hid,3hid), bqkv, Wo (hid,hid), bo, g1, b1, W1 (hid,ffn), bi1, W2 (ffn,hid), bi2, g2, b2."""
    Wqkv: torch.Tensor
    bqkv: torch.Tensor
    Wo: torch.Tensor
    bo: torch.Tensor
    g1: torch.Tensor
    b1: torch.Tensor
    W1: torch.Tensor
    bi1: torch.Tensor
    W2: torch.Tensor
    bi2: torch.Tensor
    g2: torch.Tensor
    b2: torch.Tensor

    @staticmethod
    def from_dict(p: dict, device) -> "EncoderWeights":
        return EncoderWeights(**{k: p[k].to(device=device, dtype=torch.float16).contiguous() for k in
                                 ("Wqkv", "bqkv", "Wo", "bo", "g1", "b1", "W1", "bi1", "W2", "bi2", "g2", "b2")})


class BertEncoder:
    """Forward-only encoder.  Per layer five kernel launches:
    QKV GEMM+bias -> block-masked attention reading Q/K/V straight out of the fused QKV activation and
    writing merged heads -> out-proj GEMM+bias+residual+LayerNorm -> FFN1 GEMM+bias+GELU ->
    FFN2 GEMM+bias+residual+LayerNorm (seven with `fuse_layernorm=False`: the two LayerNorms as kernels of their
    own after GEMMs with the bias + residual epilogue).  The block index is built once per mask.
    The tensor `forward` returns is one of the encoder's own buffers: it holds the result until the next forward
    pass (or graph replay) of this encoder; clone it to keep it longer."""

    def __init__(self, layers: List[EncoderWeights], head_num: int, eps: float = 1e-12, gelu: str = "erf",
                 block_m: int = 64, block_n: int = 64, fuse_layernorm: bool = True):
        """`gelu` names the feed-forward activation: "erf" (BERT), "tanh" (GPT-2 `new_gelu`) or "relu" (T5)."""
        self.fuse_layernorm = bool(fuse_layernorm)
        if gelu not in ("erf", "tanh", "relu"):
            raise _lib.StofError(f"encoder: unknown activation {gelu!r}")
        self.layers = layers
        self.head_num = head_num
        self.eps = eps
        self.gelu = gelu
        self.block_m, self.block_n = block_m, block_n
        self._index = None
        self._bufs = {}
        self._io = {}

    def set_mask(self, mask: torch.Tensor):
        """mask: (1 or B, S, S) 0/1; only mask[0] defines the block index, as in the reference."""
        self._index = get_sparse_storage(mask, self.block_m, self.block_n)[1:]
        return self._index

    def set_index(self, index):
        """index: (full_row_ptr, full_col_idx, part_row_ptr, part_col_idx, part_block_mask, load_row_ptr, load_col_idx)."""
        self._index = tuple(index)

    def _buf(self, name, shape, device):
        key = (name, tuple(shape), str(device))
        if key not in self._bufs:
            self._bufs[key] = torch.empty(shape, dtype=torch.float16, device=device)
        return self._bufs[key]

    # hidden-state buffers in rotation: while a GEMM writes one, the previous one is still its residual input and the one
    # before that may be the caller's view of the last result
    _STATES = 3

    def _activations(self, hidden):
        """(qkv, ctx, ffn intermediate, hidden states) of this input's shape, made once."""
        B, S, hid = hidden.shape
        key = (B, S, hid, self.layers[0].W1.shape[1], hidden.device)
        io = self._io.get(key)
        if io is None:
            dev = hidden.device
            states = tuple(self._buf(f"y{i}", (B, S, hid), dev) for i in range(self._STATES))
            io = self._io[key] = (self._buf("qkv", (B, S, 3 * hid), dev), self._buf("ctx", (B, S, hid), dev),
                                  self._buf("inter", (B, S, key[3]), dev), states)
        return io

    def _run(self, hidden, decoder):
        if self._index is None:
            raise _lib.StofError(f"{type(self).__name__}: call set_mask() or set_index() first")
        return (_lib._native or _lib.native()).stack(self.layers, hidden, *self._activations(hidden), *self._index[:5], self.block_m, self.block_n,
                                                     self.head_num, self.eps, EPILOGUES[self.gelu], self.fuse_layernorm, decoder)

    def forward(self, hidden: torch.Tensor) -> torch.Tensor:
        return self._run(hidden, False)

    __call__ = forward

    def capture(self, hidden: torch.Tensor):
        """Records one forward pass on `hidden` (a tensor the caller keeps and refills in place) into a CUDA graph and returns
        `replay() -> output tensor` (the output buffer is reused by every replay).  Two eager passes run first so that every
        buffer, the attention plan and its balanced schedule exist: a captured pass allocates nothing and reads nothing back.
        All launches of a pass then cost one graph launch on the host."""
        if not hidden.is_cuda:
            raise _lib.StofError("capture: hidden must live on the GPU")
        dev = hidden.device
        side = torch.cuda.Stream(dev)
        side.wait_stream(torch.cuda.current_stream(dev))
        with torch.cuda.stream(side):
            self.forward(hidden)
            self.forward(hidden)
        torch.cuda.current_stream(dev).wait_stream(side)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            out = self.forward(hidden)

        def replay():
            graph.replay()
            return out
        replay.graph = graph
        return replay


def gpt2_stack(layers: List[EncoderWeights], head_num: int, eps: float = 1e-5, block_m: int = 64, block_n: int = 64) -> BertEncoder:
    """The reference's GPT-2 loop (src/benchmk_end2end.py:93-147): the same post-LN layer with the tanh-form GELU;
    the caller sets a causal mask."""
    return BertEncoder(layers, head_num, eps, "tanh", block_m, block_n)


def t5_encoder_stack(layers: List[EncoderWeights], head_num: int, eps: float = 1e-5, block_m: int = 64, block_n: int = 64) -> BertEncoder:
    """The encoder half of the reference's T5 loop (src/benchmk_end2end.py:152-208): the same layer with ReLU."""
    return BertEncoder(layers, head_num, eps, "relu", block_m, block_n)


@dataclass
class T5DecoderWeights:
    """One decoder layer: two attention sublayers (suffix _a, _c: Wqkv, bqkv, Wo, bo, g, b) and the feed-forward
    (W1, bi1, W2, bi2, g2, b2)."""
    Wqkv_a: torch.Tensor
    bqkv_a: torch.Tensor
    Wo_a: torch.Tensor
    bo_a: torch.Tensor
    g_a: torch.Tensor
    b_a: torch.Tensor
    Wqkv_c: torch.Tensor
    bqkv_c: torch.Tensor
    Wo_c: torch.Tensor
    bo_c: torch.Tensor
    g_c: torch.Tensor
    b_c: torch.Tensor
    W1: torch.Tensor
    bi1: torch.Tensor
    W2: torch.Tensor
    bi2: torch.Tensor
    g2: torch.Tensor
    b2: torch.Tensor

    @staticmethod
    def from_dict(p: dict, device) -> "T5DecoderWeights":
        names = [f.name for f in T5DecoderWeights.__dataclass_fields__.values()]
        return T5DecoderWeights(**{k: p[k].to(device=device, dtype=torch.float16).contiguous() for k in names})


class T5Decoder(BertEncoder):
    """Decoder layers of the reference's T5 loop (src/benchmk_end2end.py:230-316): masked self-attention, a second
    attention sublayer on the decoder state, and the ReLU feed-forward, each followed by residual + LayerNorm.  Per layer
    seven kernel launches (two QKV GEMMs, two attentions, two out-projections and the second FFN GEMM with the residual + LayerNorm
    epilogue, the first FFN GEMM with ReLU)."""

    def __init__(self, layers: List[T5DecoderWeights], head_num: int, eps: float = 1e-5, block_m: int = 64, block_n: int = 64):
        super().__init__(layers, head_num, eps, "relu", block_m, block_n)

    _STATES = 4

    def forward(self, hidden: torch.Tensor) -> torch.Tensor:
        return self._run(hidden, True)

    __call__ = forward
