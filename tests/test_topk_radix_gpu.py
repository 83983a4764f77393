"""Cluster radix kernel at the edges of its splits: one to eight CTAs per row, 8 / 16 / 32 keys per thread, rows that do not
fill the last chunk, and the inputs that decide how many digits are taken."""
import pytest
import torch

from oracle import moe_oracle as O
from tilelang_moe_b200 import ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,k", [(1, 1025, 9), (3, 4096, 64), (2, 4097, 4096), (200, 8200, 65), (2, 16385, 512), (150, 16384, 2048),
                                   (160, 20001, 100), (2, 32768, 2049), (1, 65537, 1), (1, 131071, 1000), (2, 131072, 4096)])
@pytest.mark.parametrize("kind", ["normal", "narrow", "ties", "const", "sorted", "nan"])
def test_radix_splits_and_digits(cuda, lib, M, N, k, kind):
    g = torch.Generator().manual_seed(N + k)
    x = torch.randn(M, N, generator=g)
    if kind == "narrow":          # one first digit for the whole row: all three digits are needed
        x = 1.0 + x * 1e-3
    elif kind == "ties":
        x = (x * 2).round() / 2   # more equal entries at the k-th place than are sorted: the column decides
    elif kind == "const":
        x.zero_()
        x[:, ::3] = -0.0
    elif kind == "sorted":
        x = x.sort(dim=1).values
    elif kind == "nan":
        x[torch.rand(M, N, generator=g) < 0.01] = float("nan")
        x[torch.rand(M, N, generator=g) < 0.01] = float("-inf")
    xd = x.to(cuda)
    i_ref = O.stable_topk(x, k)[1]
    for mode in ("B", "A", "A_renorm"):
        s, i = ops.topk_softmax(xd, k, mode=mode)
        ops.check_status(cuda)
        assert torch.equal(i.cpu(), i_ref), (M, N, k, kind, mode)
        if kind == "nan":
            continue
        full = torch.softmax(x.double(), -1)
        top = torch.gather(x, 1, i_ref).double()
        exact = {"B": torch.softmax(top, -1), "A": torch.gather(full, 1, i_ref)}
        exact["A_renorm"] = exact["B"]
        # expf and one division in fp32 on fp64 sums: below 1e-6; the renormalised scores are divided twice
        torch.testing.assert_close(s.cpu().double(), exact[mode], rtol=1e-6, atol=1e-30)


@pytest.mark.parametrize("M,N,k", [(2, 1040, 9), (300, 3000, 200), (3, 16384, 128), (64, 32768, 32), (2, 70001, 1000), (1, 131072, 4096)])
@pytest.mark.parametrize("kind", ["one value", "two values", "masked", "grid 2^-10", "grid 2^-22", "nan"])
def test_tied_entries_are_taken_in_column_order(cuda, lib, M, N, k, kind):
    """Rows whose k-th logit has many equals: found after the second digit, the third, or all of them; the first columns stay.
    Whole numbers of grid steps keep the ties exact.  (Indices decide; scores as in the test above.)"""
    g = torch.Generator().manual_seed(N - k)
    x = torch.randn(M, N, generator=g)
    if kind == "one value":
        x.fill_(-3.5)
    elif kind == "two values":
        x = torch.where(x > 1.0, 2.0, -2.0)
    elif kind == "masked":                        # fewer finite logits than k
        x[:, torch.randperm(N, generator=g)[k // 2:]] = float("-inf")
    elif kind == "grid 2^-10":
        x = 1.0 + (x * 3).round() / 1024
    elif kind == "grid 2^-22":                    # differs in the last digit only
        x = 1.0 + (x.abs() * 2).round() / (1 << 22)
    else:
        x = torch.where(x > 0.2, float("nan"), x)
    s, i = ops.topk_softmax(x.to(cuda), k, mode="A")
    ops.check_status(cuda)
    assert torch.equal(i.cpu(), O.stable_topk(x, k)[1])
    if kind != "nan":
        exact = torch.gather(torch.softmax(x.double(), -1), 1, i.cpu())
        torch.testing.assert_close(s.cpu().double(), exact, rtol=1e-6, atol=1e-30)
