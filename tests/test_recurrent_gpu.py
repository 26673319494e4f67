"""The recurrent kernel over several tokens per launch (``fused_recurrent_kda``): both state layouts, both column
splits (few and many units), token counts around the prologue block of 16, against the CPU oracle of the recurrence."""
import pytest
import torch

from openkimi_b200.synthetic import make_inputs
from tests.kda_testlib import max_rel, rel_l2, run_oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,tol", [(torch.float32, 1e-4), (torch.bfloat16, 2e-2)])
@pytest.mark.parametrize("seqs,time,heads,d,vfirst", [
    (1, 1, 1, 64, True), (3, 16, 2, 128, True), (1, 17, 3, 128, False), (2, 33, 2, 64, False),
    (170, 2, 2, 128, True), (170, 2, 2, 128, False), (300, 3, 2, 64, True), (300, 3, 2, 64, False)])
def test_tokens_in_one_launch_match_the_oracle(dtype, tol, seqs, time, heads, d, vfirst):
    from openkimi_b200 import fused_recurrent_kda

    inp = make_inputs(seqs, time, heads, d, seed=7, dtype=dtype)
    h0 = torch.randn(seqs, heads, d, d, generator=torch.Generator().manual_seed(8)) * 0.1 if seqs > 1 else None
    ref = run_oracle(inp, h0=h0)
    tr = (lambda s: s.transpose(-1, -2).contiguous()) if vfirst else (lambda s: s)
    x = {n: inp[n].cuda() for n in ("q", "k", "v", "g", "beta")}
    o, s = fused_recurrent_kda(**x, initial_state=None if h0 is None else tr(h0.cuda()), output_final_state=True,
                               A_log=inp["a_log"].cuda(), dt_bias=inp["dt_bias"].cuda(), use_qk_l2norm_in_kernel=True,
                               use_gate_in_kernel=True, use_beta_sigmoid_in_kernel=True, state_v_first=vfirst)
    assert torch.isfinite(o.float()).all()
    assert max_rel(o, ref["o"]) <= tol and rel_l2(o, ref["o"]) <= tol
    assert max_rel(tr(s), ref["ht"]) <= tol and rel_l2(tr(s), ref["ht"]) <= tol
