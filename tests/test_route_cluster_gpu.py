"""One-launch histogram / permutation at the edges of its cluster sizes and rounds, against a stable argsort (integers: exact)."""
import pytest
import torch

from tilelang_moe_b200 import ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 31, 33, 1023, 1024, 1025, 2049, 4097, 8192, 8193, 16385, 32769, 65536, 65537])
@pytest.mark.parametrize("E", [1, 9, 256, 1000, 1024, 1025])
def test_cluster_histogram(cuda, lib, n, E):
    g = torch.Generator().manual_seed(n + E)
    for dt, spread in ((torch.int32, E), (torch.int64, max(1, E // 7))):       # the second leaves experts empty
        ids = torch.randint(0, spread, (n,), generator=g).to(dt)
        counts, offsets, perm, inv = ops.route_histogram(ids.to(cuda), E)
        want = torch.bincount(ids.long(), minlength=E)
        order = torch.argsort(ids, stable=True)
        assert torch.equal(counts.cpu().long(), want)
        assert torch.equal(offsets.cpu().long(), torch.cat([torch.zeros(1, dtype=torch.long), want.cumsum(0)]))
        assert torch.equal(perm.cpu().long(), order)
        assert torch.equal(inv.cpu().long()[order], torch.arange(n))
    ops.check_status(cuda)


def test_ids_outside_the_range_are_left_out(cuda, lib):
    ids = torch.randint(0, 40, (5000,), generator=torch.Generator().manual_seed(3), dtype=torch.int32)
    ids[::17] = -1
    ids[5::19] = 40
    keep = (ids >= 0) & (ids < 40)
    counts, offsets, perm, _ = ops.route_histogram(ids.to(cuda), 40)
    assert ops.status_buffer(cuda)[0].item() == 1          # expert id outside [0, E)
    ops.status_buffer(cuda).zero_()
    want = torch.bincount(ids[keep].long(), minlength=40)
    assert torch.equal(counts.cpu().long(), want)
    n = int(offsets[-1])
    assert n == int(keep.sum())
    where = torch.nonzero(keep).view(-1)
    assert torch.equal(perm[:n].cpu().long(), where[torch.argsort(ids[keep], stable=True)])


@pytest.mark.parametrize("n", [32768, 32769, 49152, 65535])
@pytest.mark.parametrize("E", [128, 129])
def test_one_launch_or_three(cuda, lib, n, E):
    """Either side of the rule that leaves few experts of a long list to the three kernels."""
    test_cluster_histogram(cuda, lib, n, E)
