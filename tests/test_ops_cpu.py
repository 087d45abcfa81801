"""The operators' entry points around the kernels, with the kernels replaced by plain functions on the CPU."""
import pytest
import torch
import torch.autograd.forward_ad as fwAD


@pytest.fixture
def package_op(monkeypatch):
    """`ops.package_op` with stand-ins for the launches that return what the kernels' callers would get."""
    from ops import package_op as po
    merged = lambda q, *_: q.detach().transpose(1, 2).reshape(q.shape[0], q.shape[2], -1).clone()
    for name in ("rowwise_attn_full", "rowwise_attn_sliding", "rowwise_attn_mask"):
        monkeypatch.setattr(po._rowwise, name, merged)
    monkeypatch.setattr(po, "_block_attn_mask_forward", lambda q, *_: q)
    return po


def _calls(po, q, k, v):
    i = torch.zeros(2, dtype=torch.int32)
    return {"full": lambda: po.rowwise_attn_full_op(q, k, v, False), "sliding": lambda: po.rowwise_attn_sliding_op(q, k, v, False, 3),
            "mask": lambda: po.rowwise_attn_mask_op(q, k, v, False, torch.ones(4, 4)),
            "block": lambda: po.block_attn_mask_op(q, k, v, i, i, i, i, torch.ones(1, 2, 2), i, i, 2, 2, 4)}


@pytest.mark.parametrize("name", ["full", "sliding", "mask", "block"])
@pytest.mark.parametrize("which", [0, 1, 2])
def test_forward_mode_ad_is_refused(package_op, name, which):
    """The operators have no forward-mode derivative: a tangent raises, as it does in every autograd.Function without one, and is not
    dropped.  (A dual tensor does not require grad.)"""
    qkv = [torch.randn(1, 2, 4, 64) for _ in range(3)]
    with fwAD.dual_level():
        qkv[which] = fwAD.make_dual(qkv[which], torch.ones_like(qkv[which]))
        with pytest.raises(NotImplementedError):
            _calls(package_op, *qkv)[name]()


@pytest.mark.parametrize("name", ["full", "sliding", "mask", "block"])
def test_operators_outside_differentiation(package_op, name):
    """No gradient to follow: a result that does not require grad, also for inputs that do."""
    for needs in (False, True):
        q, k, v = (torch.randn(1, 2, 4, 64, requires_grad=needs) for _ in range(3))
        with torch.no_grad():
            assert not _calls(package_op, q.detach(), k, v)[name]().requires_grad
        if name != "block":
            assert not _calls(package_op, q, k, v)[name]().requires_grad
