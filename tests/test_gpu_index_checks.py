"""Index validation of the tensor paths: int32 CUDA tensors through one kernel whose answer lands in host memory, other
integer types as before; a rejected call leaves the next one unharmed, and rasterizers share no status block."""
import pytest
import torch

import photara_drender_gb300 as pdr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.int32, torch.int64, torch.int16])
@pytest.mark.parametrize("bad", [-1, 3, 2 ** 15 - 1])
def test_out_of_range_indices_raise(dtype, bad):
    dev = torch.device("cuda", 0)
    clip = torch.tensor([[-1.0, -1, 0, 1], [1, -1, 0, 1], [0, 1, 0, 1]], device=dev)
    good = torch.tensor([[0, 1, 2]], dtype=dtype, device=dev)
    many = good.repeat(1000, 1)
    many[777, 1] = bad
    r, other = pdr.Rasterizer(), pdr.Rasterizer()
    want, _ = r.forward(clip, good, (8, 8))
    attrs = torch.rand((3, 2), device=dev)
    with pytest.raises(IndexError):
        r.forward(clip, many, (8, 8))
    with pytest.raises(IndexError):
        r.interpolate_forward(attrs, many, want)
    with pytest.raises(ValueError):
        r.interpolate_backward(attrs, many, want, torch.rand((8, 8, 2), device=dev))
    with pytest.raises(IndexError):
        r.backward(clip, many, want, torch.zeros_like(want))
    for x in (r, other):
        assert torch.equal(x.forward(clip, good, (8, 8))[0], want)
    # a transposed view: not contiguous, its elements in another order
    assert torch.equal(r.forward(clip, good.t().contiguous().t(), (8, 8))[0], want)
