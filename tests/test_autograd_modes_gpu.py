"""The autograd modes the native nodes do not support are refused, not ignored."""
import pytest
import torch
import torch.autograd.forward_ad as fwd

from openkimi_b200 import KimiDeltaAttention, chunk_kda
from tests.test_call_arguments import FUSED, _inputs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("grad", [False, True])
@pytest.mark.parametrize("name", ["q", "beta", "A_log"])
def test_forward_mode_inputs_raise(name, grad):
    x = _inputs(1, 70)
    x["v"].requires_grad_(grad)
    with fwd.dual_level():
        x[name] = fwd.make_dual(x[name], torch.ones_like(x[name]))
        with pytest.raises((RuntimeError, NotImplementedError)):
            chunk_kda(**x, **FUSED)
        with torch.no_grad(), pytest.raises((RuntimeError, NotImplementedError)):
            chunk_kda(**x, **FUSED)


@pytest.mark.parametrize("grad", [False, True])
def test_forward_mode_through_the_sublayer_raises(grad):
    mod = KimiDeltaAttention(128, 1).cuda().bfloat16().requires_grad_(grad)
    x = torch.zeros(1, 70, 128, device="cuda", dtype=torch.bfloat16)
    with fwd.dual_level(), pytest.raises((RuntimeError, NotImplementedError)):
        mod(fwd.make_dual(x, torch.ones_like(x)))
