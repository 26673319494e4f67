"""The state recurrence in parallel segments (``kda_state_seg.cu``): documents that start, end and fit inside segments,
empty documents, partial chunks, initial states and final-state gradients, both state layouts, both recompute policies,
against the FP32 CUDA-core kernels of the same op, which walk every sequence whole."""
import pytest
import torch

from openkimi_b200.synthetic import make_inputs
from tests.kda_testlib import assert_rows, compare, run_device

pytestmark = pytest.mark.gpu

CASES = {
    "one_long": [2560],
    "one_ragged": [4103],
    "uneven": [0, 1, 700, 64, 3500, 0, 3, 900, 1024, 0],
    "first_long": [3000, 40, 40, 40],
    "last_long": [65, 63, 3000],
}


@pytest.mark.parametrize("name", CASES)
@pytest.mark.parametrize("vfirst,recompute", [(True, False), (False, True)])
def test_segments_match_whole_sequences(name, vfirst, recompute):
    lens = CASES[name]
    inp = make_inputs(1, sum(lens), 2, 128, seed=3, dtype=torch.bfloat16, a_lo=0.02, a_hi=1.0)  # slow decay: states last
    cu = torch.tensor([0] + lens).cumsum(0)
    gen = torch.Generator().manual_seed(5)
    h0, dht = (torch.randn(len(lens), 2, 128, 128, generator=gen) * 0.1 for _ in range(2))
    kw = dict(h0=h0, dht=dht, cu=cu, state_v_first=vfirst)
    ref = run_device(inp, fp32_math=True, **kw)
    dev = run_device(inp, disable_recompute=not recompute, **kw)
    assert_rows(compare(dev, ref, tol_max=2e-2, tol_l2=1.5e-2))


def test_forward_only_segments_match_the_saving_forward():
    from openkimi_b200 import chunk_kda

    inp = {k: v.cuda() for k, v in make_inputs(1, 4103, 2, 128, seed=4, dtype=torch.bfloat16).items()}
    args = [inp[n] for n in ("q", "k", "v", "g", "beta")]
    kw = dict(A_log=inp["a_log"], dt_bias=inp["dt_bias"], use_qk_l2norm_in_kernel=True, use_gate_in_kernel=True,
              use_beta_sigmoid_in_kernel=True, output_final_state=True, disable_recompute=True)
    with torch.no_grad():
        o, s = chunk_kda(*args, **kw)
    o2, s2 = chunk_kda(args[0].requires_grad_(True), *args[1:], **kw)
    assert torch.equal(o, o2) and torch.equal(s, s2)


@pytest.mark.parametrize("name", ["one_ragged", "first_long", "uneven"])
@pytest.mark.parametrize("recompute", [False, True])
def test_segments_with_the_fused_convolution(name, recompute):
    """The border states lie behind another workspace with the convolution, and outside it with the recompute policy."""
    import ctypes as C

    from openkimi_b200 import _lib
    from tests.test_fused_conv_gpu import _inputs, _run, _same

    lens = CASES[name]
    p, n = _lib.KdaParams(), C.c_size_t()
    p.B, p.T, p.H, p.N, p.dk, p.dv, p.dtype = 1, sum(lens), 2, len(lens), 128, 128, _lib.DTYPE_BF16
    p.NT, p.max_chunks = sum(-(-l // 64) for l in lens), max(-(-l // 64) for l in lens)
    assert _lib.load().kda_border_bytes(C.byref(p), C.byref(n)) == 0 and n.value > 0  # this size is cut into segments
    t = _inputs(1, sum(lens), 2, 128, 4, seed=13)
    gen = torch.Generator().manual_seed(14)
    t["A_log"] = torch.log(torch.empty(2).uniform_(0.02, 1.0, generator=gen))  # slow decay: states last
    kw = dict(cu=torch.tensor([0] + lens).cumsum(0), h0=torch.randn(len(lens), 2, 128, 128, generator=gen) * 0.1)
    dev = _run(t, True, disable_recompute=not recompute, **kw)
    _same(dev, _run(t, False, disable_recompute=not recompute, **kw))
    ref = _run(t, False, fp32_math=True, **kw)
    # dA_log of a head is the sum of dg softplus / sigmoid over its elements, terms of both signs.  What a rounded record moves stays in
    # the state for the n tokens of the head's memory, so n terms move alike: their sum with a standard deviation of
    # 2.5 2^-9 sqrt(n) root-sum-square(terms) (the rms of 96 heads of other seeds).  Four of them are allowed where that is
    # more than the limit of the other outputs: a head of n = 50 draws 2.5e-2 of its dA here, whichever way single records round.
    x = (t["g"].float() + t["dt_bias"].view(1, 1, 2, 128)).double()
    terms = ref["dg"].double() * torch.nn.functional.softplus(x) / torch.sigmoid(x)
    memory = 1 / (t["A_log"].double().exp() * torch.nn.functional.softplus(x).mean((0, 1, 3)))
    bound = 10 * 2.0 ** -9 * memory.clamp_min(1).sqrt() * terms.pow(2).sum((0, 1, 3)).sqrt()
    assert ((dev["dA"] - ref["dA"]).double().abs() <= bound.clamp_min(1.5e-2 * ref["dA"].double().norm())).all()
    assert_rows(compare(dev, ref, tol_max=2e-2, tol_l2=1.5e-2, names=tuple(n for n in ref if n != "dA")))
