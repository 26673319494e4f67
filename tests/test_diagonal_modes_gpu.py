"""The two ways the BF16 forward evaluates a diagonal 16 x 16 block, with the midpoint of its rows or pair by pair, each against the
CPU oracle and against the other: their Aqk and L differ by a few 2^-22 (one or two approximated exponentials and a few
FP32 roundings each) before they are rounded to BF16 records; a flipped rounding (2^-9 of an element, fewer than one in 2^9 of
them) moves the outputs by 2^-9 sqrt(2^-9) = 9e-5 relative.  And which blocks go pair by pair: those that the guard
rejects, and all with a negative limit."""
import math

import pytest
import torch

from tests.kda_testlib import assert_rows, compare, rel_l2, run_device, run_oracle
from tests.test_kda_adversarial_gpu import _guard

pytestmark = pytest.mark.gpu
H, D = 2, 128


def _inputs(T, decay, seed, batch=1):
    """Log decays (natural) given directly: q, k normalised, beta in (0, 1)."""
    gen = torch.Generator().manual_seed(seed)
    rnd = lambda *s: torch.randn(*s, generator=gen)
    unit = lambda x: x / x.norm(dim=-1, keepdim=True)
    shape = (batch, T, H, D)
    return dict(q=unit(rnd(*shape)).bfloat16(), k=unit(rnd(*shape)).bfloat16(), v=rnd(*shape).bfloat16(),
                g=(-decay(shape, gen)).bfloat16(), beta=torch.sigmoid(rnd(*shape[:-1])).bfloat16(), do=rnd(*shape).bfloat16(),
                a_log=torch.zeros(H), dt_bias=torch.zeros(H * D))


SPANS = {
    "weak": lambda s, gen: 0.05 * torch.rand(s, generator=gen),
    "eight rows at 190": lambda s, gen: (190 / 7 * math.log(2.0)) * (0.98 + 0.02 * torch.rand(s, generator=gen)),
    "eight rows at 210": lambda s, gen: (210 / 7 * math.log(2.0)) * (1.0 + 0.02 * torch.rand(s, generator=gen)),
    "sixteen rows at 228": lambda s, gen: (228 / 15 * math.log(2.0)) * (0.98 + 0.02 * torch.rand(s, generator=gen)),
    "sixteen rows at 236": lambda s, gen: (236 / 15 * math.log(2.0)) * (1.0 + 0.02 * torch.rand(s, generator=gen)),
    "one wide channel half": lambda s, gen: torch.rand(s, generator=gen) * torch.cat([torch.ones(64), torch.full((64,), 60.0)]),
    "wide": lambda s, gen: 100 * torch.rand(s, generator=gen),
    "steps": lambda s, gen: 300 * (torch.rand(s, generator=gen) < 0.05).float(),
    "none": lambda s, gen: torch.zeros(s),
}


@pytest.mark.parametrize("name", SPANS)
@pytest.mark.parametrize("T", [16, 64, 135])
def test_midpoint_and_pairs(name, T):
    inp = _inputs(T, SPANS[name], seed=7 + T)
    ref = run_oracle(inp, fused=False)
    with _guard(232.0):
        mid = run_device(inp, fused=False)
    with _guard(-1.0):
        pairs = run_device(inp, fused=False)
    for dev in (mid, pairs):
        assert_rows(compare(dev, ref, tol_max=2e-2, tol_l2=7e-3, abs_escape=5e-5, names=("o", "ht")))
    assert rel_l2(mid["o"], pairs["o"]) <= 4 * 9e-5


@pytest.mark.parametrize("T", [16, 64, 135])
@pytest.mark.parametrize("rise", [0.02, 0.5])
def test_rising_gate_by_pairs(T, rise):
    """Single growing steps (log decays above zero) leave G not monotone; over a chunk it still falls."""
    decay = lambda s, gen: torch.where(torch.rand(s, generator=gen) < 0.2, torch.tensor(-rise), 2 * rise * torch.rand(s, generator=gen))
    inp = _inputs(T, decay, seed=11 + T)
    assert_rows(compare(run_device(inp, fused=False), run_oracle(inp, fused=False), tol_max=2e-2, tol_l2=7e-3, names=("o", "ht")))


@pytest.mark.parametrize("decay", [0.05, 40.0])
@pytest.mark.parametrize("T", [64, 1031])
def test_negative_limit_and_rejected_blocks_go_pair_by_pair(decay, T):
    """Two channels (one per half) carry no q and k.  Where their gate rises, every block is evaluated pair by pair, and nothing
    else changes: a negative limit, and the limit of a wide gate, have to give the bits of that run."""
    inp = _inputs(T, lambda s, gen: decay * torch.rand(s, generator=gen), seed=23 + T, batch=4)
    for n in ("q", "k"):
        inp[n][..., 5::64] = 0
    rising = dict(inp, g=inp["g"].clone())
    rising["g"][..., 5::64] = 0.01
    with _guard(232.0):
        want = run_device(rising, fused=False)
        kept = run_device(inp, fused=False)
    with _guard(-1.0):
        exact = run_device(inp, fused=False)
    for n in ("o", "ht"):
        assert torch.equal(exact[n], want[n]), n
        if decay > 1:  # sixteen rows span more than 232 in some channel of every block
            assert torch.equal(kept[n], want[n]), n
