"""The kernels' SiLU, its derivative, softplus and sigmoid, built on the hardware's ex2, lg2 and rcp approximations, against 64
bits.  The bounds are the approximations' documented errors (ex2 and rcp: 2 and 1 ulp, lg2 of (0.5, 2): 2^-22 absolute) and one
rounding, u = 2^-24, per operation; an argument -x log2 e carries |x| u and log2 e's own 0.22 |x| u into the exponential."""
import pytest
import torch

pytestmark = pytest.mark.gpu
U = 2.0**-24


def _grid():
    return torch.cat([torch.linspace(-80, 80, 20001), torch.linspace(-2, 2, 4999), torch.logspace(-30, 0, 500),
                      -torch.logspace(-30, 0, 500)])


def test_silu_and_its_derivative():
    from openkimi_b200.modules import short_convolution

    x = _grid()[:, None].expand(-1, 4).reshape(1, -1, 4).contiguous().cuda().requires_grad_(True)  # one tap of 1: y = silu(x)
    y = short_convolution(x, torch.ones(4, 1, 1, device="cuda"))
    y.sum().backward()
    r = x.detach().double()
    s = torch.sigmoid(r)
    # product, rcp and sum, ex2 and its argument
    assert ((y.double() - r * s).abs() <= (r * s).abs() * (8 + 1.25 * r.abs()) * U).all()
    # the same error of s once in s and once in x s (1 - s), three roundings after it
    assert ((x.grad.double() - s * (1 + r * (1 - s))).abs() <= s * (1 + r.abs()) * (12 + 1.25 * r.abs()) * U).all()


def test_softplus_of_the_decay_gate():
    """One token with k = 0: the state leaves as exp(-softplus(g + dt_bias)) times one."""
    from openkimi_b200 import chunk_kda

    H = 40
    gen = torch.Generator().manual_seed(1)
    g = torch.linspace(-40, 60, H * 128).view(1, 1, H, 128).bfloat16().cuda()
    bias = (torch.rand(H * 128, generator=gen) * 2 - 1).cuda()
    z = torch.zeros_like(g)
    _, s = chunk_kda(z, z, z, g, torch.zeros(1, 1, H, device="cuda").bfloat16(), A_log=torch.zeros(H, device="cuda"), dt_bias=bias,
                     initial_state=torch.ones(1, H, 128, 128, device="cuda"), output_final_state=True, use_gate_in_kernel=True)
    x = (g.float().view(-1) + bias).double()
    sp = torch.nn.functional.softplus(x, threshold=1000)
    err = (-s[0, :, :, 0].reshape(-1).double().log() - sp).abs()
    # the logarithm, its sum and product; sum, gate and exponent; 2^x
    assert (err <= (2.0**-22 * 0.6932 + 2 * U) + sp * 4.25 * U + 4 * U).all(), (err / (1e-7 + sp * U)).max()


def test_sigmoid_of_the_norm_gate():
    """One row of ones, an eps that adds nothing: the weight's gradient is the sigmoid in FP32, within the four ulp its kernel claims."""
    from openkimi_b200 import FusedRMSNormGated

    mod = FusedRMSNormGated(128, eps=1e-30).cuda()
    x = torch.ones(1, 128, device="cuda", dtype=torch.bfloat16)
    gates = torch.linspace(-86, 86, 128 * 64).bfloat16().view(64, 1, 128).cuda()
    for gate in gates:
        mod.weight.grad = None
        mod(x, gate).backward(x)
        want = torch.sigmoid(gate[0].double())
        assert ((mod.weight.grad.double() - want).abs() <= want * 8 * U).all()
