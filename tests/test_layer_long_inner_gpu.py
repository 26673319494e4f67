"""The sublayer's rank gradients when their inner dimension (the tokens) is cut into pieces."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_gradient_of_two_halves(dtype):
    """Sequences are independent, so a batch's weight gradients are the sums of its halves' (which are short enough not to be cut)."""
    from openkimi_b200 import KimiDeltaAttention
    from tests.kda_testlib import rel_l2

    torch.manual_seed(5)
    mod = KimiDeltaAttention(256, 2).cuda().to(dtype)
    x = torch.randn(32, 2048, 256, device="cuda").bfloat16()

    def grads(part):
        mod.zero_grad(set_to_none=True)
        with torch.autocast("cuda", torch.bfloat16):
            mod(part).square().sum().backward()
        return {k: p.grad.double() for k, p in mod.named_parameters()}

    whole, a, b = grads(x), grads(x[:16]), grads(x[16:])
    tol = 1e-3 if dtype == torch.float32 else 1e-2
    for k in whole:
        assert rel_l2(whole[k], a[k] + b[k]) < tol, k
