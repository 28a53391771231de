"""Host side of ops/wgrad.py: what is refused before a kernel is launched."""
import os

import pytest
import torch

from switchml_b200.ops import wgrad


def test_column_sums_takes_device_memory_only():
    with pytest.raises(AssertionError):
        wgrad.column_sums(torch.zeros(4, 8, dtype=torch.bfloat16))


@pytest.mark.gpu
def test_column_sums_takes_contiguous_bf16_matrices_only():
    dy = torch.zeros(16, 32, dtype=torch.bfloat16, device="cuda")
    for bad in (dy.float(), dy.t(), dy[:, :8], dy.view(2, 8, 32)):
        with pytest.raises(AssertionError):
            wgrad.column_sums(bad)


def test_layer_without_its_extension(monkeypatch, tmp_path):
    """Where the native autograd node can be neither loaded nor built, the one in Python takes its place: the same
    outputs and gradients as nn.Linear."""
    monkeypatch.setattr(wgrad, "_NODE", None)
    monkeypatch.setattr(wgrad, "_lib", lambda: None)
    monkeypatch.setattr(wgrad, "library_path", lambda name: str(tmp_path / name))
    monkeypatch.setenv("PATH", str(tmp_path))  # no compiler
    with pytest.warns(UserWarning, match="torch_switchml_linear"):
        node = wgrad._node()
    assert os.listdir(tmp_path) == []
    torch.manual_seed(0)
    plain = torch.nn.Linear(24, 16)
    grad = torch.zeros(16, 24)
    plan = node.Plan(grad, None, lambda dy, x: grad.copy_(dy.float().t() @ x.float()))
    results = []
    for f in (plain, lambda x: node.fused_linear(x, plain.weight, plain.bias, plan)):
        plain.zero_grad()
        x = torch.linspace(-1, 1, 2 * 5 * 24).view(2, 5, 24).requires_grad_()
        y = f(x)
        y.backward(torch.linspace(-2, 1, y.numel()).view(y.shape))
        results.append((y.detach(), x.grad, plain.bias.grad.clone(), plain.weight.grad))
    for got, want in zip(results[1][:3], results[0][:3]):
        assert torch.allclose(got, want, rtol=1e-5, atol=1e-5)
    assert results[1][3] is None  # the plan's buffer is the gradient
    assert float((grad - results[0][3]).norm()) < 1e-2 * float(results[0][3].norm())  # operands in bf16


@pytest.mark.gpu
@pytest.mark.parametrize("bias", [True, False])
def test_attached_layer_without_its_extension(monkeypatch, bias):
    import switchml_b200 as sml
    monkeypatch.setattr(wgrad, "_NODE", wgrad._PythonNode)
    ctx = sml.Context.get_instance()
    assert ctx.start(sml.make_config("cuda", mode="float_sum", launch="inline", symm_heap_mb=16))
    try:
        plain = torch.nn.Linear(64, 128, bias=bias, device="cuda")
        layer = wgrad.FusedWgradLinear(64, 128, bias=bias, device="cuda")
        layer.load_state_dict(plain.state_dict())
        layer.attach(ctx)
        x = torch.randn(40, 64, device="cuda")
        for module in (plain, layer):
            with torch.autocast("cuda", dtype=torch.bfloat16):
                y = module(x)
            y.backward(torch.linspace(-1, 1, y.numel(), device="cuda").view(y.shape).to(y.dtype))
            wgrad.wait_pending()
        for name, p in layer.named_parameters():
            want = dict(plain.named_parameters())[name].grad
            assert p.grad.dtype == want.dtype and float((p.grad - want).norm()) <= 1e-2 * float(want.norm())
    finally:
        ctx.stop()
