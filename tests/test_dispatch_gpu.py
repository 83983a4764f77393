"""Edges of the dispatch rules and entry points of the grouped GEMM and the fused router."""
import pytest
import torch

from tilelang_moe_b200 import kernels, ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,k,H,I,E,dtype", [(1, 1, 64, 8, 1, torch.bfloat16), (5, 3, 72, 24, 4, torch.float16),
                                             (700, 2, 256, 264, 9, torch.bfloat16), (3000, 2, 200, 64, 70, torch.float16),
                                             (4100, 1, 128, 512, 300, torch.bfloat16)])
def test_grouped_gemm_in_one_call(cuda, lib, T, k, H, I, E, dtype):
    """moe_grouped_gemm_routed against its parts called one by one: the same bits, int32 and int64 ids, on a second stream
    and replayed from a graph with other inputs."""
    g = torch.Generator().manual_seed(T + I)
    X = torch.randn(T, H, generator=g).to(dtype).to(cuda)
    W = (torch.randn(E, I, H, generator=g) * 0.05).to(dtype).to(cuda)
    ids = torch.rand(T, E, generator=g).argsort(1)[:, :k].contiguous().to(cuda)

    def parts(X, ids):
        _, offs, perm, _ = ops.route_histogram(ids, E, want_inv=False)
        xs = ops.gather_rows(X, perm, div=k)
        return ops.grouped_gemm_sorted(ops.GEMM_PLAIN, xs, W, offs, dst_rows=perm).view(T, k, I)

    want = parts(X, ids)
    assert torch.equal(kernels.grouped_gemm(X, W, ids), want)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        y = kernels.grouped_gemm(X, W, ids.int())
        static_X, static_ids = X.clone(), ids.clone()
    torch.cuda.current_stream().wait_stream(side)
    torch.cuda.synchronize()
    assert torch.equal(y, want)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = kernels.grouped_gemm(static_X, W, static_ids)
    static_X.copy_(X.flip(0))
    static_ids.copy_(ids.flip(0))
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(out, want.flip(0))
    ops.check_status(cuda)
