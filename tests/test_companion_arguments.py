"""Arguments of the sublayer's companion kernels: sizes that do not belong together and rows off a 16-byte boundary."""
import pytest
import torch

from openkimi_b200 import FusedRMSNormGated, ShortConvolution


def test_mismatched_sizes_raise():
    x = torch.zeros(2, 3, 128)
    with pytest.raises(ValueError, match="weight of shape"):
        FusedRMSNormGated(64)(x, x)
    with pytest.raises(ValueError, match="gate of shape"):
        FusedRMSNormGated(128)(x, x[:1])
    conv = ShortConvolution(128, 4)
    conv.weight = torch.nn.Parameter(torch.zeros(64, 1, 4))
    with pytest.raises(ValueError, match="filter of shape"):
        conv(x)


def test_norm_gate_entry_points_refuse_unaligned_rows():
    """Refused ahead of any launch, so addresses that are never read stand in for the tensors."""
    from openkimi_b200 import _lib

    lib, at = _lib.load(), 4096
    for bad in range(3):
        x, gate, y = (at + (2 if i == bad else 0) for i in range(3))
        assert lib.kda_norm_gate_fwd(x, gate, at, y, None, 4, 128, 1e-6, _lib.DTYPE_BF16, None) == 5
    for bad in range(5):
        x, gate, dy, dx, dgate = (at + (8 if i == bad else 0) for i in range(5))
        assert lib.kda_norm_gate_bwd(x, gate, at, dy, dx, dgate, at, at, 8, 4, 128, 1e-6, _lib.DTYPE_F32, None) == 5


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_norm_gate_of_unaligned_views(dtype):
    """Contiguous views that start anywhere in a buffer give what their copies give."""
    mod = FusedRMSNormGated(128).cuda()
    buf = torch.randn(3, 1 + 5 * 128, device="cuda").to(dtype)
    x, gate, dy = (row[1:].view(5, 128) for row in buf)
    out = []
    for a, g, d in ((x, gate, dy), (x.clone(), gate.clone(), dy.clone())):
        a, g = a.detach().requires_grad_(True), g.detach().requires_grad_(True)
        y = mod(a, g)
        out.append((y.detach(), *torch.autograd.grad(y, (a, g, mod.weight), d)))
    assert all(torch.equal(a, b) for a, b in zip(*out))


@pytest.mark.gpu
def test_tensors_on_another_device_raise():
    x = torch.zeros(2, 128, device="cuda")
    with pytest.raises(RuntimeError, match="gate on cuda"):
        FusedRMSNormGated(128).cuda()(x, x.cpu())
    with pytest.raises(RuntimeError, match="weight on cuda"):
        FusedRMSNormGated(128)(x, x)
    with pytest.raises(RuntimeError, match="weight on cuda"):
        ShortConvolution(128, 4)(x[None])
