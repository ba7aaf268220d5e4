"""Autograd behaviour of the fused model-side operators, their kernels replaced by plain PyTorch."""
import pytest
import torch
import torch.nn.functional as F


def _xent(logits, labels, grad_scale):
    keep = labels >= 0
    loss = F.cross_entropy(logits, labels.clamp(min=0), reduction="none") * keep
    d = logits.softmax(-1) - F.one_hot(labels.clamp(min=0), logits.shape[1])
    logits.copy_(d * keep[:, None] * grad_scale)
    return loss


@pytest.fixture
def case(monkeypatch):
    from dmuon_b200.ops import model_ops

    monkeypatch.setattr(model_ops, "softmax_xent_", _xent)
    torch.manual_seed(0)
    h, w = torch.randn(12, 8, requires_grad=True), torch.randn(20, 8, requires_grad=True)
    y = torch.randint(0, 20, (12,))
    y[::5] = -100
    plain = torch.autograd.grad(F.cross_entropy(F.linear(h, w), y, ignore_index=-100), (h, w))
    return h, w, lambda: model_ops._LinearXent.apply(h, w, y, 5, -100), plain


def _same(got, want, factor=1.0):
    for a, b in zip(got, want):
        assert torch.allclose(a, b * factor, atol=1e-6)


def test_linear_cross_entropy_batched_walk(case):
    h, w, loss, plain = case
    factors = torch.tensor([1.0, -2.0, 0.5])
    got = torch.autograd.grad(loss(), (h, w), grad_outputs=factors, is_grads_batched=True)
    for i, f in enumerate(factors):
        _same([t[i] for t in got], plain, f)


def test_linear_cross_entropy_derivative_of_a_factor_on_the_loss(case):
    h, w, loss, plain = case
    s = torch.tensor(3.0, requires_grad=True)
    got = torch.autograd.grad(loss() * s, (h, w), create_graph=True)
    _same(got, plain, 3.0)
    want = sum(t.sum() for t in plain)
    assert torch.allclose(torch.autograd.grad(sum(t.sum() for t in got), s)[0], want, atol=1e-5)


def test_linear_cross_entropy_leaves_packed_tensors_alone(case):
    h, w, loss, plain = case
    packed = []

    def pack(t):
        packed.append(t)
        return t

    with torch.autograd.graph.saved_tensors_hooks(pack, lambda t: t):
        out = loss() * 3.0
    before = [t.clone() for t in packed]
    _same(torch.autograd.grad(out, (h, w)), plain, 3.0)
    assert all(torch.equal(a, b) for a, b in zip(packed, before))


@pytest.mark.parametrize("frozen", [0, 1])
def test_linear_cross_entropy_of_one_argument_and_several_walks(case, frozen):
    h, w, loss, plain = case
    (h, w)[frozen].requires_grad_(False)
    out = loss() * 2.0
    for keep in (True, True, False):
        _same(torch.autograd.grad(out, (h, w)[1 - frozen], retain_graph=keep), plain[1 - frozen:2 - frozen], 2.0)
