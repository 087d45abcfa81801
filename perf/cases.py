"""Timed cases of the framework: what its users have it do, through the public entry points, over the sizes they do it at.

Six kinds of work, each with the options that are used in earnest:

  attention   block-masked attention on a block index made once per mask: the drop-in operator `block_attn_mask_op` (overwrites q)
              or `block_attention` into an output of its own
  rowwise     the row-wise operators (full, sliding, caller's mask; causal or not)
  compaction  `get_sparse_storage`: dense mask -> block index, fp16 or fp32 masks
  layernorm   bias + LayerNorm
  gemm_ln     GEMM + bias + LayerNorm
  mlp         GEMM + bias + GELU -> GEMM
  encoder     forward passes of the encoder stacks (erf GELU, tanh GELU, ReLU) and of the decoder stack

Everything is forward-only and fp16 (masks also fp32), as the operators are.
"""
import math
import os
import sys

import torch

sys.path.insert(0, os.path.join(os.getcwd(), "sc25-stof-ad_b200"))

import stof_b200  # noqa: E402
from ops.package_op import (block_attn_mask_op, rowwise_attn_full_op, rowwise_attn_mask_op,  # noqa: E402
                            rowwise_attn_sliding_op)
from triton_template.add_layernorm import triton_batched_bias_layernorm  # noqa: E402
from triton_template.gemm_add_layernorm import triton_matmul_bias_layernorm  # noqa: E402
from triton_template.gemm_gemm import triton_matmul_batch  # noqa: E402
from util.masks import get_sparse_storage  # noqa: E402

HEAD = 64


def listed():
    return [
        # one request of a small model: a 256-token sequence, +-1 block of 64 around the diagonal, the operator in place
        {"name": "attention 1x12x256 sliding", "kind": "attention", "batch": 1, "heads": 12, "seq": 256, "block": 64, "mask": "sliding", "inplace": True},
        # a middling batch with a mask that is not block-aligned (band + global tokens + scattered keys) and a length that
        # leaves half a key tile over
        {"name": "attention 4x12x1120 scattered", "kind": "attention", "batch": 4, "heads": 12, "seq": 1120, "block": 32, "mask": "scattered", "inplace": False},
        # the headline: BigBird blocks at batch 16, 2048 tokens
        {"name": "attention 16x12x2048 bigbird", "kind": "attention", "batch": 16, "heads": 12, "seq": 2048, "block": 64, "mask": "bigbird", "inplace": False},
        # long sequences with a dilated window and one global block
        {"name": "attention 8x16x4096 dilated", "kind": "attention", "batch": 8, "heads": 16, "seq": 4096, "block": 64, "mask": "dilated", "inplace": False},
        # prefill of a generating model: causal attention over the whole prompt, merged-head result
        {"name": "rowwise 8x12x1024 causal", "kind": "rowwise", "variant": "full", "batch": 8, "heads": 12, "seq": 1024, "causal": True, "window": 0},
        # the index of one short mask (a mask that changes from request to request)
        {"name": "compaction 1x512 fp16", "kind": "compaction", "batch": 1, "seq": 512, "block_m": 32, "block_n": 32, "dtype": "fp16", "mask": "scattered"},
        # the index of a batch of long fp32 masks, as mask generators of a training script leave them
        {"name": "compaction 8x4096 fp32", "kind": "compaction", "batch": 8, "seq": 4096, "block_m": 64, "block_n": 64, "dtype": "fp32", "mask": "scattered"},
        # bias + LayerNorm over the rows of a large batch
        {"name": "layernorm 8x4096x1024", "kind": "layernorm", "batch": 8, "rows": 4096, "hidden": 1024},
        # a feed-forward block on a ragged number of rows
        {"name": "mlp 3x333x768", "kind": "mlp", "batch": 3, "rows": 333, "hidden": 768, "inner": 3072},
        # one short request through a 12-layer encoder: 60 launches, latency is what counts
        {"name": "encoder 12L 1x128x768", "kind": "encoder", "model": "bert", "layers": 12, "batch": 1, "seq": 128, "hidden": 768, "mask": "sliding"},
        # an ordinary serving batch through the same encoder
        {"name": "encoder 12L 8x1024x768", "kind": "encoder", "model": "bert", "layers": 12, "batch": 8, "seq": 1024, "hidden": 768, "mask": "bigbird"},
        # the largest: a 24-layer encoder on 64 sequences of 4096 tokens
        {"name": "encoder 24L 64x4096x1024", "kind": "encoder", "model": "bert", "layers": 24, "batch": 64, "seq": 4096, "hidden": 1024, "mask": "bigbird"},
    ]


def _log(rng, lo, hi, step=1):
    """A multiple of `step` from lo to hi, spread over the logarithm."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))) / step)) * step))


def draw(rng):
    kind = rng.choice(["attention", "attention", "rowwise", "compaction", "layernorm", "gemm_ln", "mlp", "encoder", "encoder"])
    if kind == "attention":
        mask = rng.choice(["sliding", "bigbird", "dilated", "scattered"])
        block = rng.choice([16, 32, 64]) if mask == "scattered" else 64
        return {"kind": kind, "batch": _log(rng, 1, 16), "heads": rng.choice([8, 12, 16]), "seq": _log(rng, 256, 4096, block), "block": block,
                "mask": mask, "inplace": rng.random() < 0.5}
    if kind == "rowwise":
        variant = rng.choice(["full", "sliding", "mask"])
        return {"kind": kind, "variant": variant, "batch": _log(rng, 1, 16), "heads": rng.choice([8, 12, 16]), "seq": _log(rng, 128, 2048, 16),
                "causal": rng.random() < 0.7, "window": rng.choice([32, 64, 100, 256]) if variant == "sliding" else 0}
    if kind == "compaction":
        bm, bn = rng.choice([16, 32, 64, 128]), rng.choice([16, 32, 64, 128])
        return {"kind": kind, "batch": _log(rng, 1, 8), "seq": _log(rng, 256, 4096, max(bm, bn)), "block_m": bm, "block_n": bn,
                "dtype": rng.choice(["fp16", "fp32"]), "mask": rng.choice(["scattered", "bigbird"] if bm == bn == 64 else ["scattered"])}
    if kind == "layernorm":
        return {"kind": kind, "batch": _log(rng, 1, 16), "rows": _log(rng, 64, 4096), "hidden": rng.choice([256, 512, 768, 1000, 1024, 1536, 2048])}
    if kind == "gemm_ln":
        return {"kind": kind, "batch": _log(rng, 1, 16), "rows": _log(rng, 64, 4096), "inner": rng.choice([512, 768, 1024, 3072, 4096]),
                "hidden": rng.choice([512, 768, 1024])}
    if kind == "mlp":
        hidden = rng.choice([512, 768, 1024])
        return {"kind": kind, "batch": _log(rng, 1, 16), "rows": _log(rng, 64, 4096), "hidden": hidden, "inner": rng.choice([2, 4]) * hidden}
    return {"kind": kind, "model": rng.choice(["bert", "bert", "gpt2", "t5", "t5_decoder"]), "layers": _log(rng, 1, 12), "batch": _log(rng, 1, 16),
            "seq": _log(rng, 128, 2048, 64), "hidden": rng.choice([512, 768, 1024]), "mask": rng.choice(["sliding", "bigbird", "causal"])}


# ------------------------------------------------------------------------------------------
# masks: (S, S) booleans from a CPU generator
# ------------------------------------------------------------------------------------------
def _mask(recipe, seq, seed):
    i = torch.arange(seq)
    if recipe == "causal":
        return i[:, None] >= i[None, :]
    g = torch.Generator().manual_seed(seed)
    if recipe == "scattered":
        # element-granular: a band, a few global tokens, and keys strewn over a tile next to the diagonal
        on = (i[:, None] - i[None, :]).abs() <= 32
        on[:24] = True
        on[:, :24] = True
        tiles = seq // 32
        t = torch.arange(tiles).repeat_interleave(200)
        nb = (torch.arange(tiles) + 5 * torch.arange(tiles) % 7 - 3).clamp(0, tiles - 1).repeat_interleave(200)
        on[t * 32 + torch.randint(0, 32, t.shape, generator=g), nb * 32 + torch.randint(0, 32, t.shape, generator=g)] = True
        return on
    nb = -(-seq // 64)
    b = torch.arange(nb)
    d = (b[:, None] - b[None, :]).abs()
    if recipe == "sliding":
        on = d <= 1
    elif recipe == "dilated":
        on = (d <= 4) & (d % 2 == 0)
        on[0] = True
        on[:, 0] = True
    else:                               # bigbird: 3 sliding + 2 global blocks + 3 random blocks per row beside them
        on = d <= 1
        on[:2] = True
        on[:, :2] = True
        r = min(3, nb)
        on[b.repeat_interleave(r), (torch.rand(nb, nb, generator=g) + on.float()).argsort(1)[:, :r].reshape(-1)] = True
    return on.repeat_interleave(64, 0).repeat_interleave(64, 1)[:seq, :seq]


def _mask_tensor(recipe, seq, seed, dtype=torch.float16):
    return _mask(recipe, seq, seed).cuda().to(dtype).unsqueeze(0)


def _keys(case):
    """(query, key) pairs that the mask of a case admits."""
    if case["kind"] == "rowwise":
        return int(_row_mask(case, 0).sum())
    return int(_mask(case["mask"], case["seq"], 0).sum())


def _row_mask(case, seed):
    i = torch.arange(case["seq"])
    on = torch.ones(case["seq"], case["seq"], dtype=torch.bool)
    if case["variant"] == "mask":
        on = _mask("scattered", case["seq"], seed)
    elif case["variant"] == "sliding":
        on = i[None, :] > i[:, None] - case["window"]
    return on & (i[None, :] <= i[:, None]) if case["causal"] else on


# ------------------------------------------------------------------------------------------
# what a user's program holds before the call
# ------------------------------------------------------------------------------------------
def prepare(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)

    def normal(*shape, scale=1.0, shift=0.0):
        return (torch.randn(*shape, generator=g, device="cuda", dtype=torch.float16) * scale + shift)

    kind = case["kind"]
    if kind in ("attention", "rowwise"):
        shape = (case["batch"], case["heads"], case["seq"], HEAD)
        s = {"case": case, "q": normal(*shape), "k": normal(*shape), "v": normal(*shape)}
        if kind == "attention":
            s["index"] = get_sparse_storage(_mask_tensor(case["mask"], case["seq"], seed), case["block"], case["block"])[1:]
            s["out"] = torch.empty_like(s["q"])
        elif case["variant"] == "mask":
            s["row_mask"] = _mask_tensor("scattered", case["seq"], seed)[0]
        return s
    if kind == "compaction":
        mask = _mask_tensor(case["mask"], case["seq"], seed, torch.float16 if case["dtype"] == "fp16" else torch.float32)
        return {"case": case, "mask": mask.expand(case["batch"], -1, -1).contiguous()}
    if kind == "layernorm":
        h = case["hidden"]
        return {"case": case, "x": normal(case["batch"], case["rows"], h), "bias": normal(h, scale=0.1), "weight": normal(h, scale=0.1, shift=1.0),
                "bias_ln": normal(h, scale=0.1)}
    if kind == "gemm_ln":
        k, n = case["inner"], case["hidden"]
        return {"case": case, "a": normal(case["batch"], case["rows"], k), "w": normal(1, k, n, scale=0.02).expand(case["batch"], k, n),
                "bias": normal(n, scale=0.1)}
    if kind == "mlp":
        h, n = case["hidden"], case["inner"]
        return {"case": case, "a": normal(case["batch"], case["rows"], h), "b": normal(h, n, scale=0.02), "d": normal(n, h, scale=0.02),
                "bias": normal(n, scale=0.1)}
    h, f = case["hidden"], 4 * case["hidden"]

    def attention_weights(suffix, ln):
        return {"Wqkv" + suffix: normal(h, 3 * h, scale=0.02), "bqkv" + suffix: normal(3 * h, scale=0.02), "Wo" + suffix: normal(h, h, scale=0.02),
                "bo" + suffix: normal(h, scale=0.02), ln[0]: normal(h, scale=0.1, shift=1.0), ln[1]: normal(h, scale=0.1)}

    def feed_forward():
        return {"W1": normal(h, f, scale=0.02), "bi1": normal(f, scale=0.02), "W2": normal(f, h, scale=0.02), "bi2": normal(h, scale=0.02),
                "g2": normal(h, scale=0.1, shift=1.0), "b2": normal(h, scale=0.1)}

    heads = h // HEAD
    if case["model"] == "t5_decoder":
        layers = [stof_b200.T5DecoderWeights(**attention_weights("_a", ("g_a", "b_a")), **attention_weights("_c", ("g_c", "b_c")), **feed_forward())
                  for _ in range(case["layers"])]
        model = stof_b200.T5Decoder(layers, heads)
    else:
        layers = [stof_b200.EncoderWeights(**attention_weights("", ("g1", "b1")), **feed_forward()) for _ in range(case["layers"])]
        if case["model"] == "gpt2":
            model = stof_b200.gpt2_stack(layers, heads)
        elif case["model"] == "t5":
            model = stof_b200.t5_encoder_stack(layers, heads)
        else:
            model = stof_b200.BertEncoder(layers, heads)
    model.set_mask(_mask_tensor(case["mask"], case["seq"], seed))
    return {"case": case, "model": model, "hidden": normal(case["batch"], case["seq"], h)}


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "attention":
        block = case["block"]
        if case["inplace"]:
            return block_attn_mask_op(s["q"], s["k"], s["v"], *s["index"], block, block, 4)
        return stof_b200.block_attention(s["q"], s["k"], s["v"], s["out"], *s["index"], block, block)
    if kind == "rowwise":
        if case["variant"] == "full":
            return rowwise_attn_full_op(s["q"], s["k"], s["v"], case["causal"])
        if case["variant"] == "sliding":
            return rowwise_attn_sliding_op(s["q"], s["k"], s["v"], case["causal"], case["window"])
        return rowwise_attn_mask_op(s["q"], s["k"], s["v"], case["causal"], s["row_mask"])
    if kind == "compaction":
        return get_sparse_storage(s["mask"], case["block_m"], case["block_n"])
    if kind == "layernorm":
        return triton_batched_bias_layernorm(s["x"], s["bias"], s["weight"], s["bias_ln"])
    if kind == "gemm_ln":
        return triton_matmul_bias_layernorm(s["a"], s["w"], s["bias"])
    if kind == "mlp":
        return triton_matmul_batch(s["a"], s["b"], s["d"], s["bias"])
    return s["model"](s["hidden"])


def work(case):
    """Inputs read once, outputs written once; the flops of the admitted (query, key) pairs and of the matrix products."""
    kind = case["kind"]
    if kind in ("attention", "rowwise"):
        tokens = case["batch"] * case["heads"] * case["seq"]
        return {"bytes": 4 * tokens * HEAD * 2, "flops": 4.0 * HEAD * case["batch"] * case["heads"] * _keys(case)}
    if kind == "compaction":
        on = _mask(case["mask"], case["seq"], 0)
        bm, bn, s = case["block_m"], case["block_n"], case["seq"]
        share = on.view(s // bm, bm, s // bn, bn).float().mean((1, 3))
        partial, full = int(((share > 0) & (share < 1)).sum()), int((share == 1).sum())
        return {"bytes": case["batch"] * s * s * (2 if case["dtype"] == "fp16" else 4) + partial * bm * bn * 2 + 8 * (partial + full) + 12 * (s // bm + 1), "flops": 0}
    rows = case["batch"] * (case["seq"] if kind == "encoder" else case["rows"])
    h = case["hidden"]
    if kind == "layernorm":
        return {"bytes": 2 * rows * h * 2 + 3 * h * 2, "flops": 8.0 * rows * h}
    if kind == "gemm_ln":
        k = case["inner"]
        return {"bytes": 2 * (rows * k + k * h + rows * h + h), "flops": 2.0 * rows * k * h}
    if kind == "mlp":
        n = case["inner"]
        return {"bytes": 2 * (2 * rows * h + 2 * h * n + n), "flops": 4.0 * rows * h * n}
    sublayers = 2 if case["model"] == "t5_decoder" else 1
    weights = case["layers"] * (sublayers * 4 + 8) * h * h
    attention = 4.0 * HEAD * case["batch"] * (h // HEAD) * _keys(case) * sublayers * case["layers"]
    return {"bytes": 2 * (weights + 2 * rows * h), "flops": 2.0 * rows * weights + attention}


def tolerance(case):
    kind = case["kind"]
    if kind == "compaction":
        return "exact"
    if kind == "encoder":
        # fp16 activations between the operators: each layer rounds some ten times at 2^-11, and the errors add up over the layers
        return {"rel": 6e-3, "max": 0.1}
    # one or two roundings to fp16 (2^-11 = 4.9e-4 of a value), probabilities or an intermediate in fp16, sums in fp32
    return {"rel": 1e-3, "max": 2e-2}
