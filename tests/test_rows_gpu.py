"""GPU tests of the input-side convolution (layers with one pair per output row) on inputs that do not stay in L2."""
import pytest
import torch

from warpconvnet_b200._native import check_device_status
from warpconvnet_b200.nn.functional.sparse_conv import sparse_conv_rows_fused

from conftest import rel_l2

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _children(n, K, g):
    """Destination rows of ``n`` parents with one to three children each, at offsets of their own, in parent order."""
    has = torch.rand(K, n, generator=g, device=DEV).argsort(0) < torch.randint(1, 4, (n,), generator=g, device=DEV)
    place = (has.T.reshape(-1).cumsum(0) - 1).view(n, K).T
    return torch.where(has, place, -1).int().contiguous(), int(has.sum())


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("n,c_in,c_out,K", [(113664, 256, 96, 8), (113665, 256, 96, 8), (140000, 256, 48, 8), (240000, 96, 128, 8), (90001, 256, 192, 7)])
def test_groups_of_row_tiles(n, c_in, c_out, K, dtype):
    """All chunks of offsets over one group of row tiles before the next: whole groups, a last one of one tile, runs of a chunk
    that not every multiprocessor has a tile of, a last chunk of fewer offsets; every row against a matrix product per offset."""
    g = torch.Generator(device=DEV).manual_seed(n)
    dst, n_out = _children(n, K, g)
    x = torch.randn(n, c_in, generator=g, device=DEV).to(dtype)
    w = (torch.randn(K, c_in, c_out, generator=g, device=DEV) * c_in ** -0.5).to(dtype)
    want = torch.zeros(n_out, c_out, device=DEV)
    for k in range(K):
        rows = (dst[k] >= 0).nonzero()[:, 0]
        want[dst[k, rows].long()] = x[rows].float() @ w[k].float()
    got = sparse_conv_rows_fused(x, w, dst, n_out)
    check_device_status(DEV)
    # (fp32 sums, rounded once: half a unit in the last place of 16 bits)
    assert rel_l2(got.float().cpu().numpy(), want.cpu().numpy()) < {torch.float16: 5e-4, torch.bfloat16: 4e-3}[dtype]
    assert (got.float() - want).abs().max() < {torch.float16: 1e-2, torch.bfloat16: 6e-2}[dtype]


def test_rows_are_not_fetched_again_for_every_chunk():
    """256 -> 96 channels read a matrix of 205 MB in eight chunks: a row must take no longer than one of 41 MB, which stays in
    L2.  (With all rows between a chunk and the next a row took a quarter longer, in groups it takes a fifth less.)"""
    g = torch.Generator(device=DEV).manual_seed(0)
    per_row = []
    for n in (80000, 400000):
        dst, n_out = _children(n, 8, g)
        x = torch.randn(n, 256, generator=g, device=DEV).half()
        w = torch.randn(8, 256, 96, generator=g, device=DEV).half()
        times = []
        for _ in range(8):
            torch.cuda._sleep(400000)
            start, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            start.record()
            sparse_conv_rows_fused(x, w, dst, n_out)
            end.record()
            torch.cuda.synchronize()
            times.append(start.elapsed_time(end))
        per_row.append(sorted(times[2:])[2] / n)
    assert per_row[1] < per_row[0]
