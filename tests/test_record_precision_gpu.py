"""The records of the BF16 forward that are computed in FP32 and rounded once, against 64-bit sums of the same stored rows: the
diagonal 16 x 16 blocks of Aqk, and T.  An FP32 value with a relative error e rounds to another BF16 number than the exact one
in about 2 e / 2^-7.5 of all cases, so the share of entries that differ measures the error before the rounding, far
below what the outputs show."""
import ctypes as C

import pytest
import torch

pytestmark = pytest.mark.gpu
CH, D = 64, 128


def _records(q, k, v, g, beta, scale, guard=232.0, flags=0, a_log=None):
    """kda_fwd with a workspace of our own; its records Aqk, T [n, 64, 64], G, q^, k^ [n, 64, 128], beta [n, 64], n = chunk * H + head."""
    from openkimi_b200 import _lib

    B, T, H, _ = q.shape
    NT = B * (T // CH)
    p = _lib.KdaParams(B=B, T=T, H=H, dk=D, dv=D, N=B, NT=NT, dtype=_lib.DTYPE_BF16, flags=flags, scale=scale, guard_span=guard)
    o, status = torch.empty_like(v), torch.zeros(1, dtype=torch.int32, device="cuda")
    for n, t in dict(q=q, k=k, v=v, g=g, beta=beta, o=o, status=status, A_log=a_log).items():
        setattr(p, n, None if t is None else t.data_ptr())
    size = C.c_size_t()
    assert _lib.load().kda_workspace_bytes(C.byref(p), C.byref(size), None) == 0
    ws = torch.empty(size.value, dtype=torch.uint8, device="cuda")
    p.workspace, p.workspace_bytes = ws.data_ptr(), size.value
    _lib.check(_lib.load().kda_fwd(C.byref(p), None), "kda_fwd")
    torch.cuda.synchronize()
    assert int(status) == 0
    n, at, off = NT * H, {}, 0
    for name, nbytes in (("W", CH * D * 2), ("U", CH * D * 2), ("Aqk", CH * CH * 2), ("Qt", CH * D * 2), ("Kh", CH * D * 2), ("gamC", D * 4), ("Tm", CH * CH * 2),
                         ("S0", D * D * 2), ("Gc", CH * D * 4), ("Qn", CH * D * 2), ("Kn", CH * D * 2), ("aux", 3 * CH * 4)):
        at[name] = ws[off:off + n * nbytes].view(torch.float32 if name in ("gamC", "Gc", "aux") else torch.bfloat16).view(n, -1)
        off = (off + n * nbytes + 255) // 256 * 256
    core = lambda x: x.view(n, 8, 8, 8, 8).transpose(2, 3).reshape(n, CH, CH)               # core matrices of 8 x 8
    row = torch.arange(CH, device="cuda")[:, None]
    c4 = torch.arange(D // 4, device="cuda")[None]
    G = at["Gc"].view(n, CH, D // 4, 4).gather(2, (c4 ^ (row & 7))[None, :, :, None].expand(n, -1, -1, 4)).view(n, CH, D)
    c8 = torch.arange(8, device="cuda")[None]
    rows = lambda x: x.view(n, 2, CH, 8, 8).gather(3, (c8 ^ (row & 7))[None, None, :, :, None].expand(n, 2, -1, -1, 8)).view(n, 2, CH, 64).transpose(1, 2).reshape(n, CH, D)
    return core(at["Aqk"]), core(at["Tm"]), G, rows(at["Qn"]), rows(at["Kn"]), at["aux"].view(n, 3, CH)[:, 2]


def _inputs(T, H, seed, gate):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    rnd = lambda *s: torch.randn(*s, generator=gen, device="cuda")
    unit = lambda x: (x / x.norm(dim=-1, keepdim=True)).bfloat16()
    shape = (1, T, H, D)
    decay = gate * torch.nn.functional.softplus(rnd(*shape))
    return unit(rnd(*shape)), unit(rnd(*shape)), rnd(*shape).bfloat16(), (-decay).bfloat16(), torch.sigmoid(rnd(*shape[:-1])).bfloat16()


def _blocks(x):  # [n, 64, ...] -> [4 n, 16, ...]
    return x.reshape(-1, 16, *x.shape[2:])


def _diagonal(x):  # [n, 64, 64] -> the diagonal blocks [4 n, 16, 16]
    n = len(x)
    return torch.stack([x[:, 16 * b:16 * b + 16, 16 * b:16 * b + 16] for b in range(4)], 1).reshape(4 * n, 16, 16)


def _differ(got, exact, mask):
    """Share of the masked entries that are not the rounded exact ones; those below 2^-100 aside (exponentials flush at 2^-126)."""
    seen = mask & (exact.abs() >= 2.0 ** -100)
    return float((got != exact.float().bfloat16())[seen].float().mean())


def _pair_sums(x, y, G):
    """sum_d x_i y_j 2^(G_i - G_j) over blocks of 16 rows, in 64 bits (i >= j)."""
    out = torch.empty(len(x), 16, 16, dtype=torch.float64, device="cuda")
    for b in range(0, len(x), 512):
        xs, ys, g = x[b:b + 512].double(), y[b:b + 512].double(), G[b:b + 512].double()
        for i in range(16):
            e = torch.exp2((g[:, i:i + 1] - g).clamp_max(0))
            out[b:b + 512, i] = torch.einsum("nd,njd,njd->nj", xs[:, i], ys, e)
    return out


LOW, STRICT = (torch.ones(16, 16, dtype=torch.bool).tril(d) for d in (0, -1))


@pytest.mark.parametrize("guard", [232.0, -1.0])
@pytest.mark.parametrize("gate", [0.01, 1.0, 5.0, 9.0, 12.0, 40.0])
def test_diagonal_blocks(gate, guard):
    """Spans of sixteen rows from 0.2 to 1100, blocks on both sides of the guard.  FP32 multiply-adds differ in 4e-5 to 1.2e-4 of
    the entries of Aqk and 9e-5 to 1.8e-4 of T (700 000 entries: the counts spread by a tenth); operands of 22 bits in
    3e-4 and 4e-4, exponentials that flush before their product does in 1e-2."""
    q, k, v, g, beta = _inputs(20480, 4, 3, gate)
    A, T, G, qn, kn, be = _records(q, k, v, g, beta, D ** -0.5, guard)
    exact = _pair_sums(_blocks(qn), _blocks(kn), _blocks(G)) * (D ** -0.5)
    L = _pair_sums(_blocks(kn), _blocks(kn), _blocks(G)).tril(-1)
    exact_t = torch.linalg.inv(torch.eye(16, dtype=torch.float64, device="cuda") + _blocks(be).double()[:, :, None] * L)
    differ = _differ(_diagonal(A), exact, LOW.cuda()), _differ(_diagonal(T), exact_t, STRICT.cuda())
    print(gate, guard, differ)
    assert differ[0] <= 2e-4 and differ[1] <= 2.5e-4, differ


@pytest.mark.parametrize("common,limits", [(0.0, (8e-5, 1.1e-4, 1.5e-4)), (0.5, (8e-5, 2.6e-4, 3.7e-4)), (1.5, (8e-4, 1.9e-3, 2e-3))])
def test_inverse(common, limits):
    """Without a gate L is a product of BF16 rows, so all of T is the inverse in FP32.  `common`: how much the keys of a chunk share;
    the limits, for the diagonal blocks and the two levels of products below them, lie above the shares that FP32
    multiply-adds show (5e-5, 8e-5, 1.2e-4; 5e-5, 2.0e-4, 3.2e-4; 5e-4, 1.5e-3, 1.6e-3 over a million entries and more) and for
    alike keys below those of operands of 22 bits (3.3e-4, 4.1e-4; 2.3e-3, 2.5e-3)."""
    q, k, v, g, beta = _inputs(65536, 4, 5, 0.0)
    kf = k.float() + common * k.float().view(1, -1, CH, 4, D)[:, :, :1].expand(-1, -1, CH, -1, -1).reshape(k.shape)
    k = (kf / kf.norm(dim=-1, keepdim=True)).bfloat16()
    _, T, _, _, kn, be = _records(q, k, v, g, beta, D ** -0.5)
    differ = [0.0, 0.0, 0.0]
    index = torch.arange(CH, device="cuda")
    level = torch.where(index[:, None] // 16 == index // 16, 0, torch.where(index[:, None] // 32 == index // 32, 1, 2))
    for b in range(0, len(T), 1024):
        kb, lower = kn[b:b + 1024].double(), torch.ones(CH, CH, dtype=torch.bool, device="cuda").tril(-1)
        exact = torch.linalg.inv(torch.eye(CH, dtype=torch.float64, device="cuda") + be[b:b + 1024].double()[:, :, None] * (kb @ kb.transpose(1, 2)).tril(-1))
        for x in range(3):
            differ[x] += _differ(T[b:b + 1024], exact, lower & (level == x)) / (len(T) / 1024)
    print(common, differ)
    assert all(d <= m for d, m in zip(differ, limits)), differ
