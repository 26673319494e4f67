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
