"""Performance cases of the MoE layer path: routing, grouped GEMM, the fused layer and the mHC blocks around it.

Every case goes through the entry points a user calls (`tilelang_moe_b200.kernels`, and `tilelang_moe_b200.ops` for the
fused router and for mHC weights that are split once).  Five kinds of work, told apart by `case["op"]`:

  topk    kernels.topk_softmax(logits, k, mode)                        fp32 logits -> scores, int64 indices
  gemm    kernels.grouped_gemm(X, W, expert_indices)                   16-bit X and W, one or k experts per row
  layer   kernels.FusedMoETileLang(...).forward(x, weights)            the whole shared + routed layer
  router  ops.router_topk_softmax(x, Wr, k)                            router GEMM with top-k and softmax
  mhc     ops.mhc_pre, then ops.mhc_post                               the blocks on either side of the layer
"""
import math

import torch

from tilelang_moe_b200 import kernels, ops

DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16}


def listed():
    return [
        # routing of one small batch over 128 experts: a single short launch, so the call itself is what counts
        dict(name="topk_small", op="topk", M=320, N=128, k=6, mode="B"),
        # routing of a prefill batch over 256 experts, softmax over all of them first (the layer's convention)
        dict(name="topk_prefill", op="topk", M=16384, N=256, k=8, mode="A"),
        # the same kind of rows in bulk: a million tokens, bound by reading the logits
        dict(name="topk_bulk", op="topk", M=1048576, N=128, k=6, mode="B"),
        # selection from very many candidates with a large k: the radix path
        dict(name="topk_radix", op="topk", M=64, N=32768, k=2048, mode="B"),
        # expert GEMM with two experts per token on small experts: routing tables and launches weigh as much as the math
        dict(name="gemm_small", op="gemm", T=4096, k=2, H=1024, I=256, E=8, dtype="bf16"),
        # expert GEMM on the experts of a large model held by one of eight GPUs, fp16, one expert per row, ragged groups
        dict(name="gemm_large", op="gemm", T=8192, k=1, H=7168, I=2048, E=32, dtype="fp16"),
        # a decode step of a few sequences through a small layer with a shared expert: launches and latency
        dict(name="layer_decode_small", op="layer", B=8, S=1, H=2048, I=512, E=8, shared=1, k=2, dtype="bf16", routing="weight"),
        # a decode step through many mid-sized experts, a few rows each: every touched expert's weights are read once
        dict(name="layer_decode", op="layer", B=32, S=1, H=4096, I=1536, E=128, shared=0, k=8, dtype="fp16", routing="weight"),
        # one sequence through the small layer: prefill of 1024 tokens, 8 routed experts and a shared one
        dict(name="layer_small", op="layer", B=1, S=1024, H=2048, I=512, E=8, shared=1, k=2, dtype="bf16", routing="weight"),
        # prefill through the largest layer, 256 experts with a Zipf(1.1) load: the benchmark's own workload
        dict(name="layer_prefill", op="layer", B=1, S=8192, H=7168, I=2048, E=256, shared=0, k=8, dtype="bf16", routing="zipf"),
        # router of the largest layer on a long batch: a skinny GEMM with the selection behind it
        dict(name="router_large", op="router", T=16384, H=7168, E=256, k=8, dtype="bf16"),
        # mHC blocks around the layer on a long batch: bound by reading and writing the residual streams
        dict(name="mhc_large", op="mhc", T=8192, hidden=4096, hc=4),
    ]


def _log_int(rng, lo, hi, step=1):
    """A whole number in [lo, hi], spread over its logarithm, a multiple of `step`."""
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return max(lo, min(hi, int(round(v / step)) * step))


def draw(rng):
    op = rng.choice(["topk", "topk", "gemm", "layer", "layer", "router", "mhc"])
    if op == "topk":
        mode = rng.choice(["B", "A", "A_renorm"])
        if rng.random() < 0.6:      # experts of a layer: a few hundred at most, any number of tokens
            N = rng.choice([8, 16, 60, 64, 100, 128, 160, 256, 384, 512])
            return dict(op="topk", M=_log_int(rng, 1, min(1048576, (1 << 27) // N)), N=N, k=rng.randint(1, 8), mode=mode)
        N = _log_int(rng, 1040, 65536)
        return dict(op="topk", M=_log_int(rng, 1, min(4096, (1 << 25) // N)), N=N, k=_log_int(rng, 8, min(2048, N // 4)), mode=mode)
    dtype = rng.choice(["bf16", "fp16"])
    if op == "gemm":
        return dict(op="gemm", T=_log_int(rng, 1, 8192), k=rng.choice([1, 1, 2, 4]), H=_log_int(rng, 64, 7168, 8),
                    I=_log_int(rng, 64, 2048, 8), E=rng.choice([1, 4, 8, 16, 32, 64]), dtype=dtype)
    if op == "layer":
        H, I = _log_int(rng, 256, 7168, 64), _log_int(rng, 128, 2048, 8)
        E = rng.choice([8, 16, 32, 64, 128, 256])
        while 3 * E * H * I > 4_000_000_000:
            E //= 2
        T = _log_int(rng, 1, 8192)
        shared = rng.choice([0, 1, 1, 2])
        return dict(op="layer", B=1, S=T, H=H, I=I, E=E, shared=shared, k=rng.choice([1, 2, 4, 6, 8]), dtype=dtype,
                    routing="weight" if T <= 1024 else "zipf")
    if op == "router":
        return dict(op="router", T=_log_int(rng, 1, 32768), H=_log_int(rng, 512, 7168, 64),
                    E=rng.choice([8, 16, 64, 128, 160, 256]), k=rng.randint(1, 8), dtype=dtype)
    return dict(op="mhc", T=_log_int(rng, 1, 8192), hidden=_log_int(rng, 256, 4096, 8), hc=rng.choice([4, 4, 2]))


def _normal(gen, shape, dtype, std=1.0):
    return torch.empty(shape, dtype=dtype, device=gen.device).normal_(0.0, std, generator=gen)


def _zipf_logits(gen, T, E, s=1.1):
    """fp32 logits whose top-k follows a Zipf(s) popularity of the experts: log-popularity plus Gumbel noise."""
    logp = -s * torch.arange(1, E + 1, device=gen.device, dtype=torch.float32).log()
    logp = logp[torch.randperm(E, generator=gen, device=gen.device)]
    u = torch.rand(T, E, generator=gen, device=gen.device).clamp_(1e-7, 1 - 1e-6)
    return logp - (-u.log()).log()


def prepare(case, seed):
    device = torch.device("cuda", torch.cuda.current_device())
    gen = torch.Generator(device=device)
    gen.manual_seed(seed)
    op = case["op"]
    state = dict(case=case)
    if op == "topk":
        state["logits"] = _normal(gen, (case["M"], case["N"]), torch.float32)
        return state
    if op == "mhc":
        T, hc, hidden = case["T"], case["hc"], case["hidden"]
        R = 2 * hc + hc * hc
        state["residual"] = _normal(gen, (T, hc, hidden), torch.bfloat16)
        fn = _normal(gen, (R, hc * hidden), torch.float32, 1.0 / math.sqrt(hc * hidden))
        state["fn3"] = ops.mhc_split_weights(fn)                      # the weight as a program keeps it
        state["hc_scale"] = 1.0 + _normal(gen, (3,), torch.float32, 0.1)
        state["hc_base"] = _normal(gen, (R,), torch.float32, 0.1)
        state["x"] = _normal(gen, (T, hidden), torch.bfloat16)        # what the layer between the blocks hands on
        return state
    dtype = DTYPES[case["dtype"]]
    if op == "router":
        state["x"] = _normal(gen, (case["T"], case["H"]), dtype)
        state["Wr"] = _normal(gen, (case["E"], case["H"]), dtype, 1.0 / math.sqrt(case["H"]))
        return state
    if op == "gemm":
        T, k, H, I, E = (case[n] for n in ("T", "k", "H", "I", "E"))
        k = min(k, E)
        state["X"] = _normal(gen, (T, H), dtype)
        state["W"] = _normal(gen, (E, I, H), dtype, 0.02)
        ids = torch.rand(T, E, generator=gen, device=device).topk(k, dim=1).indices     # k different experts per row
        state["ids"] = ids if k > 1 else ids.reshape(T)
        return state
    B, S, H, I, E, shared, k = (case[n] for n in ("B", "S", "H", "I", "E", "shared", "k"))
    state["x"] = _normal(gen, (B, S, H), dtype)
    state["logits"] = _zipf_logits(gen, B * S, E) if case["routing"] == "zipf" else None
    router = _normal(gen, (E, H), dtype, 1.0 / math.sqrt(H))
    SI = shared * I
    shared_w = [_normal(gen, shape, dtype, 0.02) if shared else None for shape in ((SI, H), (SI, H), (H, SI))]
    routed_w = [_normal(gen, shape, dtype, 0.02) for shape in ((E, I, H), (E, I, H), (E, H, I))]
    state["weights"] = [router, *shared_w, *routed_w]
    state["layer"] = kernels.FusedMoETileLang(H, I, E, shared, k, B, S, dtype=dtype)
    return state


def run(state):
    case = state["case"]
    op = case["op"]
    if op == "topk":
        return kernels.topk_softmax(state["logits"], case["k"], mode=case["mode"])
    if op == "gemm":
        return kernels.grouped_gemm(state["X"], state["W"], state["ids"])
    if op == "layer":
        return state["layer"].forward(state["x"], *state["weights"], logits=state["logits"])
    if op == "router":
        return ops.router_topk_softmax(state["x"], state["Wr"], case["k"], mode="A")
    post_mix, comb_mix, layer_input = ops.mhc_pre(state["residual"], state["fn3"], state["hc_scale"], state["hc_base"])
    return post_mix, comb_mix, layer_input, ops.mhc_post(state["x"], state["residual"], post_mix, comb_mix)


def work(case):
    op = case["op"]
    if op == "topk":
        M, N, k = case["M"], case["N"], case["k"]
        return {"bytes": M * (4 * N + 12 * k), "flops": 2 * M * N}
    if op == "router":
        T, H, E, k = case["T"], case["H"], case["E"], case["k"]
        return {"bytes": 2 * (T * H + E * H) + 12 * T * k, "flops": 2 * T * H * E}
    if op == "mhc":
        T, hc, hidden = case["T"], case["hc"], case["hidden"]
        K, R = hc * hidden, 2 * hc + hc * hc
        # both blocks read the residual; pre reads the three bf16 parts of its weight and writes the layer input, post
        # reads x and writes the residual's successor; the mixing coefficients are written once and read once
        bytes_ = 2 * T * K * 3 + 2 * T * hidden * 2 + 2 * 3 * R * K + 4 * T * (hc + hc * hc) * 2
        return {"bytes": bytes_, "flops": 2 * T * K * (R + 2 + hc)}
    if op == "gemm":
        T, k, H, I, E = case["T"], min(case["k"], case["E"]), case["H"], case["I"], case["E"]
        touched = E * (1.0 - (1.0 - k / E) ** T)
        return {"bytes": int(2 * (T * H + touched * I * H + T * k * I) + 8 * T * k), "flops": 2 * T * k * H * I}
    T, H, I, E, shared, k = case["B"] * case["S"], case["H"], case["I"], case["E"], case["shared"], case["k"]
    touched = E * (1.0 - (1.0 - k / E) ** T)          # experts that get a row when routing is even
    router = 4 * T * E if case["routing"] == "zipf" else 2 * E * H
    flops = 6 * T * (k + shared) * H * I + (0 if case["routing"] == "zipf" else 2 * T * E * H)
    return {"bytes": int(2 * 2 * T * H + router + 2 * 3 * H * I * (touched + shared)), "flops": flops}


def tolerance(case):
    """About four times the error measured against the same path in 64 bits (2-norm, and largest value)."""
    op = case["op"]
    if op == "topk":        # measured 8e-8, 3.4e-7; indices exact, ties included
        return {"rel": 4e-7, "max": 2e-6, "differ": 0.0}
    if op == "router":      # measured 1.3e-5, and 6e-5 of the indices (logits closer than their fp32 sums)
        return {"rel": 5e-5, "max": 0.5, "differ": 3e-4}
    if op == "mhc":         # measured 1.7e-3, 3.9e-3: the rounding of the bf16 outputs
        return {"rel": 7e-3, "max": 1.6e-2}
    bf16 = case["dtype"] == "bf16"
    if op == "gemm":        # measured 1.7e-3, 3.9e-3 in bf16 and 2.1e-4, 5e-4 in fp16: the rounding of the output
        return {"rel": 7e-3, "max": 1.6e-2} if bf16 else {"rel": 8e-4, "max": 2e-3}
    # measured 2.9e-3, 2e-2 in bf16 and 3.6e-4, 2.3e-3 in fp16; with the router inside, two logits closer than their
    # fp32 sums may swap and move the values of a token's row
    swap = case["routing"] == "weight"
    return {"rel": 1.2e-2, "max": 0.5 if swap else 8e-2} if bf16 else {"rel": 1.5e-3, "max": 0.5 if swap else 1e-2}
