"""Operator API of the reference (src/ops/package_op.py), backed by the sm_100a kernels.

The row-wise operators return a new merged-head (batch, S, heads*64) tensor.
`block_attn_mask_op(q, k, v, full_row_ptr, full_col_idx, part_row_ptr, part_col_idx, part_block_mask,
load_row_ptr, load_col_idx, BLOCK_M, BLOCK_N, num_warps)` keeps the reference's contract: forward only,
positional arguments, and the returned tensor IS `q`, overwritten with the attention output
(src/ops/package_op.py:50-68).  Where the reference silently leaves a non-contiguous `q` untouched, this
version raises.
"""
import torch
from torch.autograd import Function, forward_ad

from stof_b200.attention import block_attn_mask as _block_attn_mask_forward
from stof_b200 import rowwise as _rowwise

__all__ = ['rowwise_attn_full_op', 'rowwise_attn_sliding_op', 'rowwise_attn_mask_op', 'block_attn_mask_op']


# result.shape = {batch_size, seq_len, head_num * head_size}, as in the reference (src/ops/package_op.py:10-48)
class RowWise_Attn_Full(Function):
    @staticmethod
    def forward(ctx, q, k, v, is_causal=False):
        result = _rowwise.rowwise_attn_full(q.contiguous(), k.contiguous(), v.contiguous(), is_causal)
        ctx.mark_non_differentiable(result)
        return result


class RowWise_Attn_Sliding(Function):
    @staticmethod
    def forward(ctx, q, k, v, is_causal, bandwidth):
        result = _rowwise.rowwise_attn_sliding(q.contiguous(), k.contiguous(), v.contiguous(), is_causal, bandwidth)
        ctx.mark_non_differentiable(result)
        return result


class RowWise_Attn_Mask(Function):
    @staticmethod
    def forward(ctx, q, k, v, is_causal, row_mask):
        result = _rowwise.rowwise_attn_mask(q.contiguous(), k.contiguous(), v.contiguous(), is_causal, row_mask.contiguous())
        ctx.mark_non_differentiable(result)
        return result


class Block_Attn_Mask(Function):
    @staticmethod
    def forward(ctx, q, k, v,
                full_row_ptr, full_col_idx,
                part_row_ptr, part_col_idx, part_block_mask,
                load_row_ptr, load_col_idx,
                BLOCK_M, BLOCK_N, num_warps):
        _block_attn_mask_forward(q, k, v,
                                 full_row_ptr.contiguous(), full_col_idx.contiguous(),
                                 part_row_ptr.contiguous(), part_col_idx.contiguous(), part_block_mask,
                                 load_row_ptr.contiguous(), load_col_idx.contiguous(),
                                 BLOCK_M, BLOCK_N, num_warps)
        ctx.mark_non_differentiable(q)
        return q


# The operators are forward-only: with nothing to differentiate the autograd.Function machinery (some 10 us a call) has no effect,
# and the call goes straight to the implementation.  Inside a forward-mode level it does not: a dual tensor does not require grad, and
# the Function is what refuses its tangent.
def _differentiating(q, k, v):
    return forward_ad._current_level >= 0 or (torch.is_grad_enabled() and (q.requires_grad or k.requires_grad or v.requires_grad))


def rowwise_attn_full_op(q, k, v, is_causal=False):
    if _differentiating(q, k, v):
        return RowWise_Attn_Full.apply(q, k, v, is_causal)
    return _rowwise.rowwise_attn_full(q.contiguous(), k.contiguous(), v.contiguous(), is_causal)


def rowwise_attn_sliding_op(q, k, v, is_causal, bandwidth):
    if _differentiating(q, k, v):
        return RowWise_Attn_Sliding.apply(q, k, v, is_causal, bandwidth)
    return _rowwise.rowwise_attn_sliding(q.contiguous(), k.contiguous(), v.contiguous(), is_causal, bandwidth)


def rowwise_attn_mask_op(q, k, v, is_causal, row_mask):
    if _differentiating(q, k, v):
        return RowWise_Attn_Mask.apply(q, k, v, is_causal, row_mask)
    return _rowwise.rowwise_attn_mask(q.contiguous(), k.contiguous(), v.contiguous(), is_causal, row_mask.contiguous())


def block_attn_mask_op(q, k, v, full_row_ptr, full_col_idx, part_row_ptr, part_col_idx, part_block_mask, load_row_ptr, load_col_idx,
                       BLOCK_M, BLOCK_N, num_warps):
    if _differentiating(q, k, v):
        return Block_Attn_Mask.apply(q, k, v, full_row_ptr, full_col_idx, part_row_ptr, part_col_idx, part_block_mask, load_row_ptr,
                                     load_col_idx, BLOCK_M, BLOCK_N, num_warps)
    return _block_attn_mask_forward(q, k, v, full_row_ptr.contiguous(), full_col_idx.contiguous(), part_row_ptr.contiguous(), part_col_idx.contiguous(),
                                    part_block_mask, load_row_ptr, load_col_idx, BLOCK_M, BLOCK_N, num_warps)
