"""Edges of the dispatch rules and entry points of the grouped GEMM and the fused router."""
import pytest
import torch

from oracle import moe_oracle as O
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


@pytest.mark.parametrize("T,E,k", [(1, 136, 8), (127, 256, 8), (128, 160, 6), (129, 256, 1), (255, 256, 8), (256, 200, 3),
                                   (257, 256, 8), (38000, 256, 8), (300, 128, 8), (300, 104, 8)])
@pytest.mark.parametrize("kind", ["normal", "equal", "sorted"])
def test_router_selection_in_the_epilogue(cuda, lib, T, E, k, kind):
    """One-kernel router: CTA pairs above 128 experts, single CTAs up to there; few logits above the bound (normal), all of
    them equal to it, and more above it than a row may park (ascending logits)."""
    H = 128
    g = torch.Generator().manual_seed(T + E)
    X = (torch.round(torch.randn(T, H, generator=g) * 4) / 4).bfloat16()
    W = (torch.round(torch.randn(E, H, generator=g) * 4) / 8).bfloat16()
    if kind == "equal":
        W = W[:1].repeat(E, 1)
    elif kind == "sorted":
        X[:, 0] = 8.0
        W.zero_()
        W[:, 0] = torch.arange(E).float() / 4
    X, W = X.to(cuda), W.to(cuda)
    lg = torch.full((T, E), float("nan"), device=cuda)
    for mode in ("B", "A", "A_renorm"):
        s, i = ops.router_topk_softmax(X, W, k, mode=mode, logits_out=lg, fused=True)
        ops.check_status(cuda)
        assert torch.equal(lg, ops.router_logits(X, W))
        s_ref, i_ref = O.topk_softmax(lg.cpu(), k, mode)
        assert torch.equal(i.cpu(), i_ref)
        torch.testing.assert_close(s.cpu(), s_ref, rtol=1e-6, atol=1e-30)


@pytest.mark.parametrize("T,H,E,k", [(1, 8, 1, 1), (3, 2048, 8, 2), (148, 264, 3, 3), (296, 2056, 16, 8), (297, 2048, 13, 4),
                                     (20, 3000, 32, 32), (5, 4096, 24, 6), (64, 16, 9, 2)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_few_experts_a_cta_or_a_warp_per_token(cuda, lib, T, H, E, k, dtype):
    """CUDA-core router on both sides of its rule (a CTA per token up to two per SM): inputs on a coarse grid make every
    product and sum exact in fp32, so both forms give the exact logits."""
    g = torch.Generator().manual_seed(T + H + E)
    X = (torch.round(torch.randn(T, H, generator=g) * 2) / 2).to(dtype)
    W = (torch.round(torch.randn(E, H, generator=g) * 2) / 8).to(dtype)
    lg = torch.full((T, E), float("nan"), device=cuda)
    for mode in ("B", "A", "A_renorm"):
        s, i = ops.router_topk_softmax(X.to(cuda), W.to(cuda), k, mode=mode, logits_out=lg, fused=True)
        ops.check_status(cuda)
        assert torch.equal(lg.cpu().double(), X.double() @ W.double().T)
        s_ref, i_ref = O.topk_softmax(lg.cpu(), k, mode)
        assert torch.equal(i.cpu(), i_ref)
        torch.testing.assert_close(s.cpu(), s_ref, rtol=1e-6, atol=1e-30)


@pytest.mark.parametrize("T,H,I,E,k,shared", [(1, 64, 8, 4, 2, 0), (5, 192, 40, 8, 2, 1), (31, 256, 512, 8, 2, 1), (32, 2048, 512, 8, 2, 1),
                                              (32, 320, 264, 16, 8, 0), (33, 2048, 512, 8, 2, 1), (20, 1024, 136, 6, 6, 2)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_up_gemm_of_few_rows(cuda, lib, T, H, I, E, k, shared, dtype):
    """Up to 32 tokens the layer's up GEMM holds 32 rows of A per stage: close to the oracle, and the same bits as the
    stage-by-stage layer (whose up GEMM gathers as well but does not know the rows of a group, so it takes the wide tiles
    where there are more than 32 rows in all) and, for one list of at most 32 rows, as the wide tiles on rows gathered
    beforehand."""
    from tilelang_moe_b200 import kernels, layer
    x, w = O.make_fusedmoe_inputs(1, T, H, I, E, shared, k, dtype=dtype, seed=T + I)
    names = ["router_weight", "shared_gate", "shared_up", "shared_down", "routed_gate", "routed_up", "routed_down"]
    ws = [w[n].to(cuda) if shared or not n.startswith("shared") else None for n in names]
    lg = O.router_logits(x.view(-1, H), w["router_weight"])
    m = kernels.FusedMoETileLang(H, I, E, shared, k, 1, T, dtype=dtype)
    y = m.forward(x.to(cuda), *ws, logits=lg.to(cuda))
    ref = layer.moe_forward(x.to(cuda), *ws, k, logits=lg.to(cuda))
    ops.check_status(cuda)
    assert torch.equal(y, ref)
    # the tolerances of the layer tests: 16-bit act, yk and out around fp32 sums
    exact = O.fusedmoe(x, *[w[n] if shared or not n.startswith("shared") else None for n in names], k, logits=lg)
    torch.testing.assert_close(y.float().cpu(), exact, rtol=1e-2, atol=2e-2)
    n = min(T, 32)                        # one expert list of at most 32 rows through the generic entry point
    ids = torch.randint(0, E, (n, 1), generator=torch.Generator().manual_seed(T))
    _, offs, perm, _ = O.route_histogram(ids, E)
    xs = x.view(-1, H)[:n]
    act = ops.grouped_gemm_sorted(ops.GEMM_SILU_GATE, xs.to(cuda), ws[4], offs.to(cuda), B2=ws[5], gather=perm.to(cuda))
    plain = ops.grouped_gemm_sorted(ops.GEMM_SILU_GATE, xs[perm.long()].to(cuda), ws[4], offs.to(cuda), B2=ws[5])
    ops.check_status(cuda)
    assert torch.equal(act, plain)


@pytest.mark.parametrize("T,E,k", [(1, 256, 8), (33, 256, 8), (257, 136, 7), (130, 64, 8), (31, 40, 8), (1000, 128, 3)])
@pytest.mark.parametrize("kind", ["nan", "inf", "zero rows"])
def test_router_selection_of_special_logits(cuda, lib, T, E, k, kind):
    """One-kernel router on ragged batches with NaN and infinite logits and with rows of zeros (padding tokens).  Each expert's
    weight picks columns of x, so the logits are known exactly."""
    H = 64
    g = torch.Generator().manual_seed(T + E + k)
    X = (torch.round(torch.randn(T, H, generator=g) * 4) / 4).bfloat16()
    W = torch.zeros(E, H)
    W[torch.arange(E), torch.arange(E) % 60] = 1.0 + torch.arange(E) // 60 * 0.25
    special = torch.rand(T, generator=g) < 0.4
    if kind == "nan":                             # NaN times zero: the whole row
        X[special, 3] = float("nan")
    elif kind == "inf":
        X[:, 62] = 0.0
        X[special, 62] = float("inf")
        W[:, 62] = torch.where(torch.arange(E) % 3 == 1, 1.0, -1.0)
    else:
        X[special] = 0.0
    X, W = X.to(cuda), W.bfloat16().to(cuda)
    lg = torch.full((T, E), float("nan"), device=cuda)
    for mode in ("B", "A"):
        s, i = ops.router_topk_softmax(X, W, k, mode=mode, logits_out=lg, fused=True)
        ops.check_status(cuda)
        torch.testing.assert_close(lg, ops.router_logits(X, W), rtol=0, atol=0, equal_nan=True)
        s_ref, i_ref = O.topk_softmax(lg.cpu(), k, mode)
        assert torch.equal(i.cpu(), i_ref)
        ok = lg.cpu().isfinite().all(1)
        torch.testing.assert_close(s.cpu()[ok], s_ref[ok], rtol=1e-6, atol=1e-30)
        assert kind == "inf" or s.cpu()[~ok].isnan().all()


@pytest.mark.parametrize("form", ["128", "pair", "few rows"])
def test_silu_over_its_whole_range(cuda, lib, monkeypatch, form):
    """SiLU epilogue on gates up to where exp(-g) overflows (g = -88.7; its denominator passes 2^126 at -87.3), past that, on
    infinities and NaN.  A gate is a sum of two weights, so it is exact; exp is within 2^-17, the result rounded to bf16 once."""
    if form != "few rows":
        monkeypatch.setenv("MOE_B200_GEMM_TILE_ROWS", form)
    g = torch.cat([torch.arange(-5673, -5586) / 64, torch.linspace(-87, 20, 400), torch.tensor([0.0, 1e-20, -1e-20, 300.0, 1e30]),
                   torch.tensor([-89.0, -200.0, -1e30, float("inf"), float("-inf"), float("nan")])])
    g = torch.cat([g, torch.zeros(-len(g) % 64)])
    N, K, rows = len(g), 64, 5 if form == "few rows" else 300
    hi = g.bfloat16()
    lo = torch.where(hi.isfinite(), g - hi.float(), 0.0).bfloat16()
    gate = hi.double() + lo.double()
    Wg, Wu, A = torch.zeros(1, N, K), torch.zeros(1, N, K), torch.zeros(rows, K)
    Wg[0, :, 0], Wg[0, :, 1], Wu[0, :, 0], A[:, 0], A[:, 1] = hi.float(), lo.float(), 1.0, 1.0, 1.0
    args = [t.bfloat16().to(cuda) for t in (A, Wg, Wu)]
    offs = torch.tensor([0, rows], dtype=torch.int32, device=cuda)
    gather = torch.arange(rows, dtype=torch.int32, device=cuda) if form == "few rows" else None
    y = ops.grouped_gemm_sorted(ops.GEMM_SILU_GATE, args[0], args[1], offs, B2=args[2], gather=gather).cpu().double()
    ops.check_status(cuda)
    exact = gate / (1.0 + torch.exp(-gate))
    near = gate.isfinite() & (gate >= -88.65)
    torch.testing.assert_close(y[:, near], exact[near].expand(rows, -1), rtol=2.0 ** -8, atol=0)
    far = gate.isfinite() & (gate < -88.65)
    assert far.any() and bool(((y[:, far] <= 0) & (y[:, far] > -1e-35)).all())
    assert bool((y[:, gate == float("inf")] == float("inf")).all()) and bool(y[:, ~gate.isfinite() & (gate != float("inf"))].isnan().all())


@pytest.mark.parametrize("T,H,E,k", [(7, 1016, 16, 2), (7, 1024, 16, 2), (40, 256, 9, 3), (40, 256, 8, 3), (40, 256, 17, 3)])
def test_a_cta_or_a_warp_per_token_of_short_rows(cuda, lib, T, H, E, k):
    """... and on the sides of its rule on the hidden size and the number of experts."""
    test_few_experts_a_cta_or_a_warp_per_token(cuda, lib, T, H, E, k, torch.bfloat16)


@pytest.mark.parametrize("K,N", [(64, 8), (128, 200), (192, 512)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_epilogue_of_few_and_many_rows_per_warp(cuda, lib, K, N, dtype):
    """Groups that end in warps of 1 to 32 rows, 64-row and 128-row tiles: rows stored directly and through shared memory, scattered
    and scaled.  Inputs on a coarse grid make every sum exact in fp32, so the result is its one rounding."""
    sizes = [1, 2, 15, 16, 17, 31, 32, 33, 48, 49, 0, 64, 65, 79, 80, 81, 97, 112, 113, 127, 128, 129, 145]
    E, n = len(sizes), sum(sizes)
    g = torch.Generator().manual_seed(K + N)
    A = (torch.randn(n, K, generator=g) * 2).round().clamp(-4, 4).to(dtype)
    W = ((torch.randn(E, N, K, generator=g) * 2).round().clamp(-4, 4) / 8).to(dtype)
    offs = torch.tensor([0, *sizes]).cumsum(0).int()
    dst = torch.randperm(n, generator=g).int()
    w = torch.randint(1, 9, (n,), generator=g).float() / 4
    y = torch.cat([A[a:b].float() @ W[e].float().T for e, (a, b) in enumerate(zip(offs[:-1].tolist(), offs[1:].tolist()))])
    dev = [t.to(cuda) for t in (A, W, offs, dst, w)]
    want = torch.empty(n, N, dtype=dtype)
    want[dst.long()] = y.to(dtype)
    assert torch.equal(ops.grouped_gemm_sorted(ops.GEMM_PLAIN, dev[0], dev[1], dev[2], dst_rows=dev[3]).cpu(), want)
    want[dst.long()] = (y * w[:, None]).to(dtype)
    got = ops.grouped_gemm_sorted(ops.GEMM_SCALE_SCATTER, dev[0], dev[1], dev[2], dst_rows=dev[3], row_w=dev[4])
    assert torch.equal(got.cpu(), want)
    ops.check_status(cuda)


@pytest.mark.parametrize("T,E", [(4095, 128), (4096, 128), (9472, 136), (9473, 136), (700, 64)])
def test_router_on_the_sides_of_its_rule(cuda, lib, T, E):
    """One kernel or two, as the rule picks: the same logits, so the same scores and indices."""
    g = torch.Generator().manual_seed(T)
    X, W = torch.randn(T, 64, generator=g).bfloat16().to(cuda), torch.randn(E, 64, generator=g).bfloat16().to(cuda)
    s, i = ops.router_topk_softmax(X, W, 6, mode="A")
    ops.check_status(cuda)
    for fused in (True, False):
        s2, i2 = ops.router_topk_softmax(X, W, 6, mode="A", fused=fused)
        assert torch.equal(i, i2)
        torch.testing.assert_close(s, s2, rtol=2e-6, atol=0)
