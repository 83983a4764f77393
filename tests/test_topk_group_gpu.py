"""Lane-group and lane-per-row top-k kernels at the edges of their ranges: row lengths around every lane split, all k, and
the three ways a row's entries are collected (few entries, many equal ones, too many above the bound)."""
import pytest
import torch

from oracle import moe_oracle as O
from tilelang_moe_b200 import ops

pytestmark = pytest.mark.gpu
RTOL = 1e-6   # fp32 softmax of at most 1024 terms: a few ulp of expf and of the sum, as for the other top-k kernels


def _rows(kind, M, N, g):
    x = torch.randn(M, N, generator=g)
    if kind == "ties":            # a few distinct values: more entries equal to the bound than a row may collect
        x = x.round()
    elif kind == "const":
        x.zero_()
        x[::2] = -0.0
    elif kind == "sorted":        # ascending rows: whole parts of the row lie above the bound
        x = x.sort(dim=1).values
    elif kind == "masked":        # most experts masked out
        x[torch.rand(M, N, generator=g) < 0.9] = float("-inf")
        x[:, 0] = 0.0             # one finite logit at least: a softmax over -inf alone is NaN
    elif kind == "nan":
        x[torch.rand(M, N, generator=g) < 0.02] = float("nan")
        x[torch.rand(M, N, generator=g) < 0.02] = float("inf")
    return x


@pytest.mark.parametrize("kind", ["normal", "ties", "const", "sorted", "masked", "nan"])
@pytest.mark.parametrize("N", [8, 12, 32, 36, 64, 68, 72, 128, 132, 256, 260, 512, 516, 1000, 1024])
def test_group_and_lane_kernels(cuda, lib, N, kind):
    M = 2051 if N <= 256 else 83     # the last warp's rows run past the end
    g = torch.Generator().manual_seed(N)
    x = _rows(kind, M, N, g)
    xd = x.to(cuda)
    for k in (1, 2, 3, 4, 6, 7, 8):
        for mode in ("B", "A", "A_renorm"):
            s, i = ops.topk_softmax(xd, k, mode=mode)
            if kind == "nan":        # scores of such rows are NaN or depend on inf - inf: the order is what counts
                assert torch.equal(i.cpu(), O.stable_topk(x, k)[1])
                continue
            s_ref, i_ref = O.topk_softmax(x, k, mode)
            assert torch.equal(i.cpu(), i_ref), (N, k, mode, kind)
            torch.testing.assert_close(s.cpu(), s_ref, rtol=RTOL, atol=1e-30)
    ops.check_status(cuda)


def test_padded_rows_and_both_index_types(cuda, lib):
    base = torch.randn(4100, 192, generator=torch.Generator().manual_seed(1)).to(cuda)
    for N in (24, 100, 188):
        view = base[:, 4:4 + N]                       # row stride 192, rows 16-byte aligned
        s, i64, i32 = ops.topk_softmax(view, 5, also_int32=True)
        s_ref, i_ref = O.topk_softmax(view.cpu(), 5)
        assert torch.equal(i64.cpu(), i_ref) and torch.equal(i32.cpu().long(), i_ref)
        torch.testing.assert_close(s.cpu(), s_ref, rtol=RTOL, atol=1e-30)


def test_large_row_counts_take_fewer_lanes_per_row(cuda, lib):
    x = torch.randn(262145, 68, device=cuda, generator=torch.Generator(device=cuda).manual_seed(2))
    s, i = ops.topk_softmax(x, 8)                     # four lanes per row
    s1, i1 = ops.topk_softmax(x[:262144], 8)          # eight
    assert torch.equal(i[:-1], i1)
    torch.testing.assert_close(s[:-1], s1, rtol=2 * RTOL, atol=1e-30)   # two kernels, each within RTOL of the exact scores
    rows = torch.arange(0, 262145, 997)
    s_ref, i_ref = O.topk_softmax(x[rows.to(cuda)].cpu(), 8)
    assert torch.equal(i[rows.to(cuda)].cpu(), i_ref)
    torch.testing.assert_close(s[rows.to(cuda)].cpu(), s_ref, rtol=RTOL, atol=1e-30)
