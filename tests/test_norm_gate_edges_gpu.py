"""The output gate of the RMS norm at the ends of its range: the BF16 kernels' sigmoid clamps its argument."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim", [64, 128])
def test_saturated_gates(dim):
    from openkimi_b200 import FusedRMSNormGated

    edges = torch.tensor([0.0, 30.0, -30.0, 87.0, -87.0, 100.0, -101.0, 3e38, -3e38, float("inf"), -float("inf")])
    gen = torch.Generator().manual_seed(3)
    x = torch.randn(3, dim, generator=gen).bfloat16()
    gate = edges[torch.arange(3 * dim) % edges.numel()].view(3, dim).bfloat16()
    mod = FusedRMSNormGated(dim).cuda()
    xd, gd = x.cuda().requires_grad_(True), gate.cuda().requires_grad_(True)
    y = mod(xd, gd)
    y.backward(torch.ones_like(y))
    xr = x.double()
    ref = xr * (xr.square().mean(-1, keepdim=True) + mod.eps).rsqrt() * torch.sigmoid(gate.double())
    assert torch.allclose(y.detach().cpu().double(), ref, rtol=2**-8, atol=1e-30)
    assert torch.isfinite(xd.grad).all() and torch.isfinite(gd.grad).all()
    assert mod(xd, torch.full_like(gd, float("nan"))).isnan().all()


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("rows", [1, 3, 17])
def test_no_eps(dtype, rows):
    """eps = 0: rows past the last one, which a warp holds as zeros, leave no NaN in the weight's gradient."""
    from openkimi_b200 import FusedRMSNormGated

    gen = torch.Generator().manual_seed(rows)
    x, gate, dy = (torch.randn(rows, 64, generator=gen).to(dtype) for _ in range(3))
    mod = FusedRMSNormGated(64, eps=0.0).cuda()
    mod(x.cuda(), gate.cuda()).backward(dy.cuda())
    xr = x.double()
    want = (dy.double() * torch.sigmoid(gate.double()) * xr * xr.square().mean(-1, keepdim=True).rsqrt()).sum(0)
    scale = (dy.double() * xr).abs().sum(0)
    assert ((mod.weight.grad.cpu().double() - want).abs() <= 1e-5 * scale).all()  # FP32 sums of at most 17 terms
