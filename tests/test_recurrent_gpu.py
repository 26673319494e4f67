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


@pytest.mark.parametrize("d,vfirst,seqs", [(128, True, 73), (128, True, 74), (128, False, 18), (128, False, 19), (64, True, 295),
                                           (64, True, 296), (64, False, 73), (64, False, 74)])
def test_both_sides_of_the_column_split(d, vfirst, seqs):
    """Each sequence alone (eight columns per warp) against all of them at once: the same FP32 sums, in another order for
    [dk][dv] states (64 terms a lane at most and five levels: 70 * 2^-24 = 4e-6 of the magnitudes; 1e-5 with cancellation)."""
    from openkimi_b200 import fused_recurrent_kda

    gen = torch.Generator(device="cuda").manual_seed(9)
    r = lambda *s: torch.randn(*s, generator=gen, device="cuda")
    x = {n: r(seqs, 2, 2, d) for n in ("q", "k", "v", "g")} | {"beta": r(seqs, 2, 2)}
    kw = dict(A_log=r(2) * 0.1, output_final_state=True, use_qk_l2norm_in_kernel=True, use_gate_in_kernel=True,
              use_beta_sigmoid_in_kernel=True, state_v_first=vfirst)
    h0 = r(seqs, 2, d, d) * 0.1
    o, s = fused_recurrent_kda(**x, initial_state=h0, **kw)
    for n in (0, seqs // 2, seqs - 1):
        o1, s1 = fused_recurrent_kda(**{k: v[n:n + 1] for k, v in x.items()}, initial_state=h0[n:n + 1], **kw)
        assert rel_l2(o[n:n + 1], o1) < 1e-5 and rel_l2(s[n:n + 1], s1) < 1e-5
