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


@pytest.mark.parametrize("heads,tokens", [(1, 15000), (1, 13000), (2, 13999), (3, 20003), (6, 20905), (6, 20951)])
def test_rank_gradients_around_the_line(heads, tokens):
    """Two sequences together against each alone: cut or not, with every kind of remainder.  FP32 sums over up to 42000 tokens in
    different orders: 42000 * 2^-24 = 2.5e-3 of the sum of the terms' magnitudes at the very worst, sqrt(42000) * 2^-24 = 1.2e-5
    expected; 1e-4 of the norm."""
    from openkimi_b200 import KimiDeltaAttention
    from tests.kda_testlib import rel_l2

    torch.manual_seed(tokens)
    mod = KimiDeltaAttention(128, heads).cuda()
    x, dy = (torch.randn(2, tokens, 128, device="cuda").bfloat16() for _ in range(2))

    def grads(a, d):
        mod.zero_grad(set_to_none=True)
        with torch.autocast("cuda", torch.bfloat16):
            mod(a).backward(d)
        return [mod.f_b_proj.weight.grad.double(), mod.out_gate_b.weight.grad.double()]

    whole, a, b = grads(x, dy), grads(x[:1], dy[:1]), grads(x[1:], dy[1:])
    for w, p, q in zip(whole, a, b):
        assert rel_l2(w, p + q) < 1e-4
