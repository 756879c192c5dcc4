"""argmax_rows on both sides of the line between a cluster and a CTA per row: ties (the lowest index, wherever its part of the row is worked on), rows
of nothing but -inf, rows that start at any multiple of 4 bytes, more rows than a grid has in y.  Whole numbers: equal to a linear scan."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,d,pad", [(1, 1, 0), (3, 320, 1), (64, 32767, 1), (64, 32768, 0), (65, 32768, 0), (2, 128256, 3), (64, 128257, 0), (512, 32000, 0), (70000, 37, 2)])
def test_first_maximum(rows, d, pad):
    from cactus_b200._lib import check, lib
    g = torch.Generator(device="cuda").manual_seed(rows + d)
    x = torch.randn((rows, d + pad), device="cuda", generator=g)
    x[:, d:] = 100.0                                                   # beyond the row
    first = torch.randint(0, d, (rows,), device="cuda", generator=g)
    second = torch.randint(0, d, (rows,), device="cuda", generator=g)
    at = torch.arange(rows, device="cuda")
    x[at, first] = x[at, second] = 9.0                                 # a tie
    want = torch.minimum(first, second).int()
    x[0, :d] = float("-inf")
    want[0] = 0
    out = torch.full((rows,), -1, dtype=torch.int32, device="cuda")
    check(lib().b200_argmax_rows(x.data_ptr(), (d + pad) * 4, d, rows, out.data_ptr(), torch.cuda.current_stream().cuda_stream))
    assert torch.equal(out, want)
