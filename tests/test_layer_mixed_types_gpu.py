"""Sublayer parameters of mixed types under autocast: an FP32 parameter's gradient is not rounded to BF16 because another
parameter, whose gradient comes from the same product, is BF16."""
import pytest
import torch

from openkimi_b200 import KimiDeltaAttention

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("low", [("f_b_proj",), ("f_a_proj",), ("q_proj", "v_proj"), ("out_proj", "out_gate_b", "beta_proj")])
def test_fp32_gradients_beside_bf16_parameters(low):
    torch.manual_seed(3)
    mod = KimiDeltaAttention(256, 2).cuda()
    with torch.no_grad():  # weights that are the same numbers in both types
        for p in mod.parameters():
            p.copy_(p.bfloat16())
    x, dy = (torch.randn(2, 300, 256, device="cuda").bfloat16() for _ in range(2))

    def grads():
        mod.zero_grad(set_to_none=True)
        with torch.autocast("cuda", torch.bfloat16):
            mod(x).backward(dy)
        return {n: p.grad for n, p in mod.named_parameters()}

    want = grads()
    for name in low:
        getattr(mod, name).bfloat16()
    got = grads()
    for n, g in got.items():
        bf16 = n.split(".")[0] in low
        assert g.dtype == (torch.bfloat16 if bf16 else torch.float32), n
        assert torch.equal(g, want[n].to(g.dtype)), n
