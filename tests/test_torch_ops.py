"""The torch front end without a GPU: what autograd is told about the two ops, on meta tensors."""
import pytest
import torch

from flash_attention3_b200 import torch_binding


@pytest.fixture
def qkv():
    return [torch.empty((1, h, 48, 64), dtype=torch.float16, device="meta", requires_grad=True) for h in (4, 2, 2)]


def test_attention_has_a_first_derivative(qkv):
    out = torch_binding.attention(*qkv, causal=True)
    grads = torch.autograd.grad(out.float().square().sum(), qkv)
    assert [g.shape for g in grads] == [t.shape for t in qkv]
    assert not any(g.requires_grad for g in grads)


def test_second_derivatives_are_refused(qkv):
    out = torch_binding.attention(*qkv, causal=True)
    dq, = torch.autograd.grad(out.float().square().sum(), qkv[:1], create_graph=True)
    with pytest.raises(RuntimeError, match="attention_bwd is not implemented"):
        torch.autograd.grad(dq.float().sum(), qkv)


def test_differentiating_the_ops_is_refused(qkv):
    out, lse = torch.ops.fa3b200.attention_fwd(*qkv, True, 0.125)
    assert out.requires_grad and lse.requires_grad
    for t in (out, lse):
        with pytest.raises(RuntimeError, match="attention_fwd is not implemented"):
            torch.autograd.grad(t.float().sum(), qkv[:1], retain_graph=True)
    with torch.no_grad():
        assert not torch.ops.fa3b200.attention_fwd(*qkv, True, 0.125)[0].requires_grad


def test_attention_takes_the_arguments_that_the_ops_take(qkv):
    """Numbers and flags as in the schema of the ops: what torch would turn away there is turned away."""
    for accepted in (dict(causal=1), dict(causal=None), dict(window=[3, 0]), dict(window=torch.tensor([3, 0])),
                     dict(softcap="0.5"), dict(softmax_scale=1), dict(deterministic=torch.tensor(True))):
        assert torch_binding.attention(*qkv, **accepted).shape == qkv[0].shape
    for refused in (dict(causal="x"), dict(causal=[]), dict(window=(1.5, 0)), dict(window=("1", "0")), dict(window=(1,)),
                    dict(window=None), dict(softmax_scale="0.5"), dict(softcap=None), dict(layout=3), dict(deterministic="x")):
        with pytest.raises((TypeError, ValueError, IndexError, RuntimeError)):
            torch_binding.attention(*qkv, **refused)


def test_ops_are_marked_fit_for_compilation():
    for op in (torch_binding.attention_fwd, torch_binding.attention_bwd):
        assert torch.Tag.pt2_compliant_tag in op.tags
