"""Edges of the layer kernels' tiles: one and several tiles per CTA, whole and
half column slices, one and two stages of A, unaligned optional operands (GPU).

Reference: the same BF16 operands multiplied in FP64 by torch.  Tolerances,
relative to the largest output: FP32 sums 1e-5 for K <= 256 (16 MMA steps of
2^-23 with the epilogue's roundings); the hardware tanh's 2^-11 enters the
activated column sums, where it averages to below 1e-4; the long reductions
2^-23 per MMA step and 2^-24 per split, below 5e-5 for the sizes here; BF16
outputs one rounding and the tanh, 1e-2.
"""
import pytest

from conftest import pkg

pytestmark = pytest.mark.gpu


def rel(a, b):
    return float((a.double() - b).abs().max() / b.abs().max())


@pytest.mark.parametrize("M,N,K", [(1, 256, 256), (129, 256, 256), (30000, 256, 256), (20001, 192, 256),
                                   (500, 224, 256), (20000, 160, 240), (40000, 256, 64), (20000, 64, 256)])
@pytest.mark.parametrize("zpad", [0, 1, 8])
def test_linear_tiles(cuda_device, M, N, K, zpad):
    import torch
    ops = pkg("mlp_ops")
    torch.manual_seed(M + N)
    X = torch.randn(M, K, device=cuda_device).bfloat16()
    W = (torch.randn(N, K, device=cuda_device) / K ** 0.5).bfloat16()
    b = torch.randn(N, device=cuda_device)
    zp = torch.randn(M, N + zpad, device=cuda_device).bfloat16()[:, zpad:]
    ref = X.double() @ W.double().t()
    Y32 = torch.empty(M, N, device=cuda_device)
    Z = torch.empty(M, N, device=cuda_device, dtype=torch.bfloat16)
    ops.linear(X, W, bias=b, Y32=Y32, Z=Z)
    assert rel(Y32, ref + b) < 1e-5
    assert rel(Z, ref + b) < 1e-2
    Y = torch.empty(M, N, device=cuda_device, dtype=torch.bfloat16)
    YT = torch.zeros(N, M, device=cuda_device, dtype=torch.bfloat16)
    cs = torch.ones(N, device=cuda_device)
    ops.linear(X, W, zprev=zp, Y=Y, YT=YT, colsum=cs)
    z = zp.double()
    s = torch.sigmoid(z)
    ref = ref * (s * (1 + z * (1 - s)))
    assert ops.status() == 0
    assert rel(Y, ref) < 1e-2
    assert torch.equal(YT.t(), Y)
    assert float((cs.double() - 1 - ref.sum(0)).abs().max()) < 1e-4 * float(ref.abs().sum(0).max())


def test_linear_output_over_its_input(cuda_device):
    import torch
    ops = pkg("mlp_ops")
    torch.manual_seed(3)
    X = torch.randn(20000, 256, device=cuda_device).bfloat16()
    W = (torch.randn(256, 256, device=cuda_device) / 16).bfloat16()
    Y = torch.empty_like(X)
    ops.linear(X, W, Y=Y)
    ops.linear(X, W, Y=X)
    assert ops.status() == 0
    assert torch.equal(X, Y)


@pytest.mark.parametrize("Mo,No,Kb", [(1, 32, 64), (64, 256, 64), (256, 64, 192), (130, 96, 64 * 601),
                                      (256, 256, 64 * 77)])
@pytest.mark.parametrize("cpad", [0, 1])
def test_wgrad_ring(cuda_device, Mo, No, Kb, cpad):
    import torch
    ops = pkg("mlp_ops")
    torch.manual_seed(Mo + No)
    A = torch.randn(Mo, Kb, device=cuda_device).bfloat16()
    B = torch.randn(No, Kb, device=cuda_device).bfloat16()
    C = torch.ones(Mo, No + cpad, device=cuda_device)[:, cpad:]
    ops.wgrad(A, B, C)
    assert ops.status() == 0
    assert rel(C, 1 + A.double() @ B.double().t()) < 5e-5


@pytest.mark.parametrize("M", [1, 129, 152 * 128, 152 * 128 + 1, 304 * 128 + 1, 100001])
@pytest.mark.parametrize("off", [0, 1])
def test_fused_forward_ring(cuda_device, M, off):
    """One and two CTAs per SM, one and several tiles per CTA, unaligned biases;
    the layers one by one give the same roundings, so 1e-2 only allows for a
    few activations that round the other way."""
    import torch
    ops = pkg("mlp_ops")
    torch.manual_seed(M)
    dims = [(256, 64)] + [(256, 256)] * 3 + [(64, 256)]
    W = [(torch.randn(n, k, device=cuda_device) / k ** 0.5).bfloat16() for n, k in dims]
    b = [torch.randn(n + off, device=cuda_device)[off:] for n, _ in dims]
    a = X = torch.randn(M, 64, device=cuda_device).bfloat16()
    Y = torch.full((M + 1, 64), 7.0, device=cuda_device)
    ops.forward_fused(X, [ops.pack_core(w) for w in W], b, Y=Y[:M])
    for l in range(4):
        n = torch.empty(M, 256, device=cuda_device, dtype=torch.bfloat16)
        ops.linear(a, W[l], bias=b[l], act=True, Y=n)
        a = n
    ref = torch.empty(M, 64, device=cuda_device)
    ops.linear(a, W[4], bias=b[4], Y32=ref)
    assert ops.status() == 0
    assert rel(Y[:M], ref.double()) < 1e-2
    assert bool((Y[M] == 7.0).all())


@pytest.mark.parametrize("M", [1, 63, 64, 1000, 152 * 64 * 4 + 65])
def test_head_grad(cuda_device, M):
    """Column sums: FP32 over M rows in partial sums, 1e-5 of the sum of magnitudes."""
    import torch
    ops = pkg("mlp_ops")
    torch.manual_seed(M)
    dY = torch.randn(M, 64, device=cuda_device)
    Z = torch.empty(M, 64, device=cuda_device, dtype=torch.bfloat16)
    ZT = torch.empty(64, M, device=cuda_device, dtype=torch.bfloat16)
    cs = torch.ones(64, device=cuda_device)
    ops.head_grad(dY, Z, ZT, cs)
    assert torch.equal(Z, dY.bfloat16()) and torch.equal(ZT, dY.bfloat16().t())
    d = (cs.double() - 1 - dY.double().sum(0)).abs().max()
    assert float(d) < 1e-5 * float(1 + dY.double().abs().sum(0).max())


def test_backward_takes_any_layout_of_its_gradient(cuda_device):
    import torch
    net = pkg("surrogate").MLP(torch.device(cuda_device))
    X = torch.randn(128, 64, device=cuda_device).bfloat16()
    XT = X.t().contiguous()
    dY = torch.randn(128, 64, device=cuda_device)
    out = []
    for d in (dY, dY.t().contiguous().t(), torch.cat([dY, dY], 1)[:, :64]):
        net.forward(X, keep=True)
        gW, gb = net.backward(XT, d)
        out.append(gW + gb)
    for o in out[1:]:
        for a, b in zip(out[0], o):
            assert a.shape == b.shape and a.dtype == b.dtype
            assert float((a - b).abs().max()) <= 1e-5 * float(b.abs().max()) + 1e-30
