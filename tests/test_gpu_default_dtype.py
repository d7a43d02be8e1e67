"""The network's gradients are FP32 whatever torch's default dtype is (GPU)."""
import pytest

from conftest import pkg

pytestmark = pytest.mark.gpu


@pytest.fixture
def fp64_default():
    torch = pytest.importorskip("torch")
    old = torch.get_default_dtype()
    torch.set_default_dtype(torch.float64)
    yield torch
    torch.set_default_dtype(old)


def _pass(torch, device):
    g = torch.Generator().manual_seed(5)
    X = torch.randn(256, 64, generator=g, dtype=torch.float32).to(device).bfloat16()
    dY = torch.randn(256, 64, generator=g, dtype=torch.float32).to(device)
    net = pkg("surrogate").MLP(device)
    Y = net.forward(X, keep=True).clone()
    gW, gb = net.backward(X.t().contiguous(), dY)
    net.adam(gW, gb, 1e-3)
    return [Y] + gW + gb + net.W + net.b


def test_training_step_under_fp64_default(cuda_device, fp64_default):
    torch = fp64_default
    got = _pass(torch, cuda_device)
    torch.set_default_dtype(torch.float32)
    for a, b in zip(got, _pass(torch, cuda_device)):
        assert a.dtype == b.dtype == torch.float32
        # partial sums meet by atomics: their order, not the inputs, may differ
        assert float((a - b).abs().max()) <= 1e-5 * float(b.abs().max()) + 1e-30


@pytest.mark.parametrize("bad", ["dtype", "size", "stride"])
def test_head_grad_checks_its_column_sums(cuda_device, bad):
    import torch
    ops = pkg("mlp_ops")
    dY = torch.zeros(64, 64, device=cuda_device)
    Z = torch.empty(64, 64, device=cuda_device, dtype=torch.bfloat16)
    cs = {"dtype": torch.zeros(64, device=cuda_device, dtype=torch.float64),
          "size": torch.zeros(63, device=cuda_device),
          "stride": torch.zeros(128, device=cuda_device)[::2]}[bad]
    with pytest.raises(ValueError):
        ops.head_grad(dY, Z, torch.empty_like(Z), cs)
