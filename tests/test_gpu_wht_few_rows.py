"""Batched FP32 Walsh-Hadamard transform around the number of rows up to which
a tile is a row (2^11 and 2^12: the SMs, tensor form, or twice as many): both
sides of each line, in place and not.  Tolerance: 2e-6 * max|ref| against the
FP64 transform (FP32 arithmetic over at most 12 add/sub stages)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("method,per_sm", [("tensor", 1), ("cuda", 2)])
@pytest.mark.parametrize("log2n", [11, 12])
@pytest.mark.parametrize("extra", [-1, 0, 1])
@pytest.mark.parametrize("in_place", [False, True])
def test_around_the_line(gpu, method, per_sm, log2n, extra, in_place):
    import torch

    from compmatmul_b200 import device
    rows = per_sm * torch.cuda.get_device_properties(0).multi_processor_count + extra
    g = torch.Generator(device="cuda").manual_seed(rows + log2n)
    x = torch.randn((rows, 1 << log2n), device="cuda", generator=g)
    ref, h = x.double(), 1
    while h < 1 << log2n:
        ref = ref.view(rows, -1, 2, h)
        ref = torch.stack([ref[:, :, 0] + ref[:, :, 1], ref[:, :, 0] - ref[:, :, 1]], dim=2).view(rows, -1)
        h *= 2
    y = device.wht_rows(x, method, out=x if in_place else None)
    assert (y - ref).abs().max() <= 2e-6 * ref.abs().max()
