"""Hooks and replaced forwards of the sublayer's parts run, whether they belong to one module or to all."""
import pytest
import torch
from torch.nn.modules.module import register_module_forward_hook, register_module_full_backward_hook

from openkimi_b200 import KimiDeltaAttention

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["own", "global", "backward", "forward"])
def test_parts_are_called(kind):
    torch.manual_seed(0)
    mod = KimiDeltaAttention(128, 1).cuda().bfloat16()
    x = torch.randn(1, 70, 128, device="cuda", dtype=torch.bfloat16)
    y, seen, handle = mod(x), [], None
    if kind == "own":
        mod.out_proj.register_forward_hook(lambda m, i, o: seen.append(m))
    elif kind == "global":
        handle = register_module_forward_hook(lambda m, i, o: seen.append(m))
    elif kind == "backward":
        handle = register_module_full_backward_hook(lambda m, i, o: seen.append(m))
    else:
        plain = mod.out_proj.forward
        mod.out_proj.forward = lambda i: seen.append(mod.out_proj) or plain(i)
    try:
        out = mod(x)
        out.sum().backward()
    finally:
        if handle is not None:
            handle.remove()
    assert any(m is mod.out_proj for m in seen)
    assert (out.float() - y.float()).norm() < 1e-2 * y.float().norm()
