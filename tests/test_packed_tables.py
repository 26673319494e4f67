"""Document boundaries have to lie inside the batch: the kernels read and write the rows they name."""
import pytest
import torch

from openkimi_b200 import ops


@pytest.mark.parametrize("cu,tokens", [([0, 70, 131], 130), ([-1, 130], 130), ([0, 1], 0)])
@pytest.mark.parametrize("on_host", [False, True])
def test_boundaries_outside_the_batch_raise(cu, tokens, on_host):
    cu = torch.tensor(cu)
    with pytest.raises(ValueError, match="cu_seqlens must stay within"):
        ops._packed_tables(cu, cu if on_host else None, torch.empty(1, tokens, 2, 128))


@pytest.mark.gpu
def test_boundaries_inside_the_batch():
    """The last token ends a document, or belongs to none: both are computed."""
    from openkimi_b200 import chunk_kda
    from tests.test_call_arguments import FUSED, _inputs

    x = _inputs(1, 130)
    whole, _ = chunk_kda(**x, cu_seqlens=torch.tensor([0, 70, 130], device="cuda"), **FUSED)
    part, _ = chunk_kda(**x, cu_seqlens=torch.tensor([0, 70, 100], device="cuda"), **FUSED)
    assert torch.equal(whole[:, :100], part[:, :100])
    for cu in ([0, 70, 131], [-64, 130]):
        with pytest.raises(ValueError, match="cu_seqlens must stay within"):
            chunk_kda(**x, cu_seqlens=torch.tensor(cu, device="cuda"), **FUSED)
