"""Arguments of ``chunk_kda`` and of the decoding calls that the native host path has to refuse or to honour."""
import pytest
import torch

from openkimi_b200 import chunk_kda, fused_recurrent_kda, recurrent_kda_step

pytestmark = pytest.mark.gpu
FUSED = dict(use_qk_l2norm_in_kernel=True, use_gate_in_kernel=True, use_beta_sigmoid_in_kernel=True)


def _inputs(*lead, heads=2, dim=128, dtype=torch.bfloat16):
    x = {n: torch.randn(*lead, heads, dim, device="cuda").to(dtype) for n in ("q", "k", "v", "g")}
    return dict(x, beta=torch.randn(*lead, heads, device="cuda").to(dtype), A_log=torch.zeros(heads, device="cuda"),
                dt_bias=torch.zeros(heads * dim, device="cuda"))


def test_tensors_on_another_device_raise():
    x, s = _inputs(2, 5), torch.zeros(2, 2, 128, 128, device="cuda")
    taps = [torch.zeros(256, 1, 4, device="cuda") for _ in range(3)]
    for name in ("A_log", "dt_bias"):
        bad = dict(x, **{name: x[name].cpu()})
        with pytest.raises(RuntimeError, match=name):
            chunk_kda(**bad, **FUSED)
        with pytest.raises(RuntimeError, match=name):
            fused_recurrent_kda(**bad, **FUSED)
    with pytest.raises(RuntimeError, match="initial_state"):
        chunk_kda(**x, initial_state=s.cpu(), **FUSED)
    with pytest.raises(RuntimeError, match=r"short_conv_weights\[1\]"):
        chunk_kda(**x, short_conv_weights=(taps[0], taps[1].cpu(), taps[2]), **FUSED)
    # what the call does not use may be anywhere
    y = dict(x, g=-x["g"].abs(), beta=x["beta"].sigmoid(), A_log=x["A_log"].cpu(), dt_bias=None)
    chunk_kda(**y)
    fused_recurrent_kda(**y)


def test_in_place_states_of_any_layout():
    """A state off a 16-byte boundary, or with strides of its own, is updated in place like any other."""
    x = _inputs(3)
    want = torch.randn(3, 2, 128, 128, device="cuda")
    buf = torch.empty(1 + want.numel(), device="cuda")
    off, strided = buf[1:].view(want.shape), torch.empty(3, 2, 128, 256, device="cuda")[..., ::2]
    o1, s1 = recurrent_kda_step(**x, state=want, **FUSED)
    for state in (off, strided, want.transpose(-1, -2).contiguous().transpose(-1, -2), want.clone().requires_grad_(True)):
        with torch.no_grad():
            state.copy_(want)
        o2, s2 = recurrent_kda_step(**x, state=state, inplace=True, **FUSED)
        assert torch.equal(o1, o2) and torch.equal(s1, state) and torch.equal(s1, s2)
        assert s2.data_ptr() == state.data_ptr() and not s2.requires_grad
    wide = want[:1].expand(3, -1, -1, -1).contiguous()
    o3, s3 = recurrent_kda_step(**x, state=wide, **FUSED)
    o4, s4 = recurrent_kda_step(**x, state=want[:1].expand(3, -1, -1, -1), inplace=True, **FUSED)
    assert torch.equal(o3, o4) and torch.equal(s3, s4) and not torch.equal(want[0], s4[0])


def test_a_step_needs_a_state():
    for inplace in (False, True):
        with pytest.raises(TypeError, match="state"):
            recurrent_kda_step(**_inputs(2), state=None, inplace=inplace, **FUSED)
