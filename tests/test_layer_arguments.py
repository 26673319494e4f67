"""The sublayer's native node takes its sizes from the input and the head count: inputs and parameters of other sizes, or on
another device, have to reach the composed path, which computes them or raises."""
import pytest
import torch
import torch.nn as nn

from openkimi_b200 import KimiDeltaAttention

NAMES = ("q_proj.weight", "k_proj.weight", "v_proj.weight", "q_conv.weight", "k_conv.weight", "v_conv.weight", "A_log",
         "f_a_proj.weight", "f_b_proj.weight", "dt_bias", "beta_proj.weight", "out_gate_a.weight", "out_gate_b.weight",
         "out_norm_gate.weight", "out_proj.weight")


def _parameters(mod):
    named = dict(mod.named_parameters())
    return [named[n].detach() for n in NAMES]


def test_node_takes_only_matching_tensors():
    from openkimi_b200 import _lib

    takes = _lib.host().layer_takes
    mod = KimiDeltaAttention(192, 2)
    prm, x = _parameters(mod), torch.zeros(1, 5, 192)
    assert takes(x, prm, 2)
    assert takes(x, _parameters(KimiDeltaAttention(192, 2, conv_kernel=3)), 2)
    for bad in (torch.zeros(1, 5, 184), torch.zeros(1, 5, 200), torch.zeros(5, 192), torch.zeros(1, 5, 192, device="meta")):
        assert not takes(bad, prm, 2), bad.shape
    assert not takes(x, prm, 1) and not takes(x, prm, 3) and not takes(x, prm[:-1], 2)
    for i, name in enumerate(NAMES):
        last = prm[i].shape[-1]
        for other in (prm[i].narrow(-1, 0, last - 1), torch.cat([prm[i], prm[i].narrow(-1, 0, 1)], -1), prm[i][None],
                      prm[i][:-1] if prm[i].dim() > 1 else prm[i][:0], prm[i].to("meta")):
            assert not takes(x, prm[:i] + [other] + prm[i + 1:], 2), (name, other.shape, other.device)


@pytest.mark.gpu
@pytest.mark.parametrize("width", [184, 200, 128])
def test_input_of_another_width_raises(width):
    mod = KimiDeltaAttention(192, 2).cuda()
    with torch.autocast("cuda", torch.bfloat16), pytest.raises(RuntimeError):
        mod(torch.zeros(2, 5, width, device="cuda", dtype=torch.bfloat16))


@pytest.mark.gpu
def test_parameters_of_other_sizes():
    torch.manual_seed(0)
    mod = KimiDeltaAttention(192, 2).cuda()
    x = torch.randn(2, 70, 192, device="cuda", dtype=torch.bfloat16)
    with torch.no_grad(), torch.autocast("cuda", torch.bfloat16):
        y = mod(x)
        keep = mod.out_proj
        mod.out_proj = nn.Linear(256, 320, bias=False, device="cuda")  # an output of another width is a module's right
        mod.out_proj.weight[:192] = keep.weight
        wide = mod(x)
        assert wide.shape == (2, 70, 320)
        assert (wide[..., :192].float() - y.float()).norm() < 1e-2 * y.float().norm()
        mod.out_proj = nn.Linear(248, 192, bias=False, device="cuda")
        with pytest.raises(RuntimeError):
            mod(x)
        mod.out_proj = keep
        for name, shape in (("q_conv", (128, 1, 4)), ("A_log", (3,)), ("dt_bias", (2, 64))):
            old = getattr(mod, name)
            new = nn.Parameter(torch.zeros(shape, device="cuda"))
            if name == "q_conv":
                weight, old.weight = old.weight, new
            else:
                setattr(mod, name, new)
            with pytest.raises(ValueError):
                mod(x)
            if name == "q_conv":
                old.weight = weight
            else:
                setattr(mod, name, old)
        assert torch.equal(mod(x), y)
