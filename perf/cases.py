"""Performance cases of lightop_b200: what a serving program has the framework do, through its public entry points.

Five paths, told apart by the case's ``path``:

* ``layer``   gate + fused block-INT8 expert layer (``moe.fused_experts_impl_int8``, 128x128 block scales), the framework's
              main path: decode to prefill, one GPU with all experts or one shard of an expert-parallel group
* ``channel`` the same layer in the per-channel W8A8 format
* ``stages``  the per-channel layer composed by the caller from the stand-alone operators
* ``masked``  the expert side of expert-parallel decode on the masked layout (two grouped GEMMs and the activation)
* ``linear``  the dense block-INT8 linear on bf16 input (activation quantisation + GEMM)

Sizes: the DeepSeek-V3 and Qwen3 expert shapes and the tiny shape of ``lightop_b200.synthetic.CONFIGS``, the linear and
ragged shapes of the tests, token counts from 1 to 8192.
"""
from __future__ import annotations

import math

import torch

from lightop_b200 import activation, gemm_ops, moe, quant, synthetic

# experts, top-k, hidden, intermediate
SHAPES = {
    "dsv3": (256, 8, 7168, 2048),
    "qwen3": (128, 8, 4096, 1536),
    "small": (32, 8, 1024, 384),
    "tiny": (8, 2, 256, 512),
}
# N, K of dense linears: the shapes of the tests and the shared expert's two projections at the DeepSeek-V3 widths
LINEARS = ((576, 7168), (1536, 1536), (2304, 1280), (4096, 7168), (7168, 2048))


def _layer(name, shape, M, gate="softmax", zipf=0.0, shared=False, shards=1, graph=False, path="layer"):
    case = {"path": path, "shape": shape, "M": M, "gate": gate, "zipf": zipf, "shared": shared, "shards": shards,
            "graph": graph}
    return dict(case, name=name) if name else case


def listed():
    return [
        # a layer so small that launches and host work are all there is (unit-test and draft-model sizes)
        _layer("tiny_layer", "tiny", 32),
        # interactive decode, one sequence: eight experts' weights, latency-bound
        _layer("decode_1", "dsv3", 1),
        # batched decode as serving engines run it: the step captured once and replayed as a CUDA graph
        _layer("decode_64_graph", "dsv3", 64, graph=True),
        # a mixed batch of prefill pieces and decodes, odd size, with the grouped sigmoid gate, the shared expert's output
        # added in the reduction and a routed scaling factor
        _layer("mixed_777_grouped", "dsv3", 777, gate="grouped", shared=True),
        # prefill batch, the headline workload
        _layer("prefill_4096", "dsv3", 4096),
        # prefill with skewed expert popularity: a few hot experts, many cold ones, some without tokens
        _layer("prefill_2048_zipf", "qwen3", 2048, zipf=1.2),
        # one GPU of an eight-way expert-parallel group: 32 of the 256 experts, through an expert map
        _layer("shard_8192", "dsv3", 8192, shards=8),
        # per-channel weights, prefill, odd token count
        _layer("channel_prefill_2999", "dsv3", 2999, path="channel"),
        # a program that composes the layer from the stand-alone operators
        _layer("stages_300", "qwen3", 300, path="stages"),
        # expert side of expert-parallel decode: 32 local experts, up to 128 rows each, about 20 on average
        {"path": "masked", "E": 32, "max_m": 128, "mean_m": 20, "H": 7168, "I": 2048, "name": "masked_decode"},
        # dense linear of one decoded token; N is not a multiple of the tile
        {"path": "linear", "M": 1, "N": 576, "K": 7168, "name": "linear_1"},
        # dense linear of a prefill batch
        {"path": "linear", "M": 4096, "N": 4096, "K": 7168, "name": "linear_4096"},
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.49)))))))


def draw(rng):
    path = rng.choices(("layer", "channel", "stages", "masked", "linear"), (10, 2, 2, 2, 4))[0]
    if path == "linear":
        N, K = rng.choice(LINEARS)
        return {"path": path, "M": _log_int(rng, 1, 4096), "N": N, "K": K}
    if path == "masked":
        max_m = rng.choice((64, 128, 256))
        H, I = rng.choice(((7168, 2048), (4096, 1536)))
        return {"path": path, "E": rng.choice((16, 32)), "max_m": max_m, "mean_m": _log_int(rng, 1, max_m * 3 // 4), "H": H, "I": I}
    shape = rng.choices(("dsv3", "qwen3", "small", "tiny"), (5, 3, 1, 1))[0]
    big = shape in ("dsv3", "qwen3")
    if path == "stages":
        return _layer(None, shape, _log_int(rng, 16, 2048), path=path)
    shards = 8 if path == "layer" and big and rng.random() < 0.25 else 1
    M = _log_int(rng, 1, 8192 if shards > 1 else 4096)
    grouped = shape == "dsv3" and rng.random() < 0.4
    return _layer(None, shape, M, gate="grouped" if grouped else "softmax",
                  zipf=1.2 if shape == "qwen3" and rng.random() < 0.5 else 0.0,
                  shared=rng.random() < 0.4, shards=shards, graph=path == "layer" and M <= 256 and rng.random() < 0.5, path=path)


# ------------------------------------------------------------------ inputs

def _bf16(g, *shape):
    return torch.randn(*shape, generator=g, device="cuda").to(torch.bfloat16)


def _prepare_layer(case, seed):
    E, k, H, I = SHAPES[case["shape"]]
    M, E_local = case["M"], E // case["shards"]
    g = torch.Generator(device="cuda").manual_seed(seed + 2)
    w1, w2, w1_s, w2_s = synthetic.make_weights(E_local, H, I, seed=seed, device="cuda")
    if case["path"] != "layer":
        w1_s, w2_s = synthetic.make_channel_scales(E_local, H, I, seed=seed, device="cuda")
    x, logits = synthetic.make_activations(M, H, E, seed=seed + 1, device="cuda", zipf=case["zipf"] or None)
    s = {"case": case, "x": x, "logits": logits, "w1": w1, "w2": w2, "w1_s": w1_s, "w2_s": w2_s, "k": k, "E": E,
         "bias": None, "shared": None, "map": None}
    if case["gate"] == "grouped":
        s["bias"] = torch.randn(E, generator=g, device="cuda") * 0.02      # a correction, small beside the scores' spread
    if case["shared"]:
        s["shared"] = _bf16(g, M, H)
    if case["shards"] > 1:      # this GPU holds the experts [E_local, 2 * E_local) of the group
        s["map"] = torch.full((E,), -1, dtype=torch.int32, device="cuda")
        s["map"][E_local:2 * E_local] = torch.arange(E_local, dtype=torch.int32, device="cuda")
    # the scratch a program keeps for the layer's routed rows
    s["cache13"] = torch.empty(M * k * H, dtype=torch.bfloat16, device="cuda")
    if case["graph"]:
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            _run_layer(s)
        torch.cuda.current_stream().wait_stream(side)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            s["outputs"] = _run_layer(s)
        s["graph"] = graph
    return s


def prepare(case, seed):
    path = case["path"]
    if path in ("layer", "channel", "stages"):
        return _prepare_layer(case, seed)
    g = torch.Generator(device="cuda").manual_seed(seed)
    if path == "linear":
        M, N, K = case["M"], case["N"], case["K"]
        w = torch.randint(-127, 128, (N, K), generator=g, device="cuda", dtype=torch.int8)
        w_s = torch.rand((N + 127) // 128, K // 128, generator=g, device="cuda") * 9e-3 + 1e-3
        return {"case": case, "x": _bf16(g, M, K), "w": w, "w_s": w_s}
    E, max_m, H, I = case["E"], case["max_m"], case["H"], case["I"]
    w1, w2, _, _ = synthetic.make_weights(E, H, I, seed=seed, device="cuda")
    w1_s, w2_s = synthetic.make_channel_scales(E, H, I, seed=seed, device="cuda")
    x_q, x_s = quant.per_token_quant_int8(_bf16(g, E * max_m, H))
    # rows per expert: uniform from none to twice the mean
    counts = torch.randint(0, 2 * case["mean_m"] + 1, (E,), generator=g, device="cuda").clamp_(max=max_m).to(torch.int32)
    return {"case": case, "x_q": x_q.view(E, max_m, H), "x_s": x_s.view(E, max_m, 1), "w1": w1, "w2": w2, "w1_s": w1_s,
            "w2_s": w2_s, "counts": counts,
            # the dispatcher's fixed-capacity buffers; rows beyond an expert's count are never written
            "h": torch.zeros(E, max_m, 2 * I, dtype=torch.bfloat16, device="cuda"),
            "y": torch.zeros(E, max_m, H, dtype=torch.bfloat16, device="cuda")}


# ------------------------------------------------------------------ one pass

def _route(s):
    logits, k = s["logits"], s["k"]
    if s["bias"] is not None:
        return moe.moe_fused_gate(logits, s["bias"], 8, 4, k, 0, 2.5, False)
    M = logits.shape[0]
    weights = torch.empty(M, k, dtype=torch.float32, device=logits.device)
    ids = torch.empty(M, k, dtype=torch.int32, device=logits.device)
    moe.topk_softmax(weights, ids, None, logits, True)
    return weights, ids


def _run_layer(s):
    weights, ids = _route(s)
    block = s["case"]["path"] == "layer"
    y = moe.fused_experts_impl_int8(
        s["x"], s["w1"], s["w2"], weights, ids, s["cache13"], use_int8_w8a8=True, per_channel_quant=not block,
        block_shape=[128, 128] if block else None, w1_scale=s["w1_s"], w2_scale=s["w2_s"],
        global_num_experts=s["E"], expert_map=s["map"], routed_scaling_factor=2.5 if s["bias"] is not None else 1.0,
        shared_output=s["shared"])
    return {"y": y, "weights": weights, "ids": ids}


def _run_stages(s):
    x, w1, w2, k, E = s["x"], s["w1"], s["w2"], s["k"], s["E"]
    M, H = x.shape
    I = w2.shape[2]
    block = 16 if M * k <= 16 * E else (64 if M * k <= 64 * E else 128)
    weights, ids = _route(s)
    sorted_ids, expert_ids, num_post = moe.moe_align_block_size(ids, block, E)
    config = {"BLOCK_SIZE_M": block}
    x_q, x_s = quant.per_token_quant_int8(x)
    h = torch.empty(M, k, 2 * I, dtype=torch.bfloat16, device=x.device)
    moe.moe_gemm_w8a8(x_q, w1, h, x_s, s["w1_s"].unsqueeze(-1), None, sorted_ids, expert_ids, num_post, k, config)
    a_q, a_s = activation.fuse_silu_mul_quant(h.view(M * k, 2 * I))
    rows = s["cache13"].view(M, k, H)
    moe.moe_gemm_w8a8(a_q, w2, rows, a_s, s["w2_s"].unsqueeze(-1), weights, sorted_ids, expert_ids, num_post, 1, config)
    y = torch.empty_like(x)
    moe.moe_sum(rows, y)
    return {"y": y, "weights": weights, "ids": ids}


def _run_masked(s):
    mean = s["case"]["mean_m"]
    gemm_ops.m_grouped_w8a8_gemm_nt_masked((s["x_q"], s["x_s"]), (s["w1"], s["w1_s"]), s["h"], s["counts"], mean)
    a_q, a_s = activation.fuse_silu_mul_quant_ep(s["h"], s["counts"])
    gemm_ops.m_grouped_w8a8_gemm_nt_masked((a_q, a_s), (s["w2"], s["w2_s"]), s["y"], s["counts"], mean)
    return s["y"]


def run(state):
    path = state["case"]["path"]
    if path == "linear":
        return gemm_ops.apply_w8a8_block_int8_linear(state["x"], state["w"], [128, 128], state["w_s"])
    if path == "masked":
        return _run_masked(state)
    if path == "stages":
        return _run_stages(state)
    if "graph" in state:
        state["graph"].replay()
        return state["outputs"]
    return _run_layer(state)


# ------------------------------------------------------------------ what a pass cannot do without

def _experts_hit(E, k, M, zipf):
    """Expected number of experts that receive a token."""
    if not zipf:
        return E * (1.0 - (1.0 - k / E) ** M)
    g = torch.Generator().manual_seed(0)
    logits = torch.randn(2048, E, generator=g) - zipf * torch.log(torch.arange(1, E + 1, dtype=torch.float32))
    share = torch.bincount(logits.topk(k, dim=1).indices.reshape(-1), minlength=E).double() / 2048
    return float((1.0 - (1.0 - share) ** M).sum())


def work(case):
    path = case["path"]
    if path == "linear":
        M, N, K = case["M"], case["N"], case["K"]
        return {"bytes": 2.0 * M * K + N * K + 4.0 * ((N + 127) // 128) * (K // 128) + 2.0 * M * N, "flops": 2.0 * M * N * K}
    if path == "masked":
        E, H, I = case["E"], case["H"], case["I"]
        m = min(case["mean_m"], case["max_m"])
        hit = E * 2 * case["mean_m"] / (2 * case["mean_m"] + 1)
        return {"bytes": hit * (3.0 * H * I + 4.0 * (2 * I + H)) + E * m * (H + 4.0 + 2.0 * H), "flops": 6.0 * E * m * H * I}
    E, k, H, I = SHAPES[case["shape"]]
    M, shards = case["M"], case["shards"]
    hit = _experts_hit(E, k, M, case["zipf"]) / shards
    scales = 4.0 * 3 * (H // 128) * (I // 128) if path == "layer" else 4.0 * (2 * I + H)
    io = 2.0 * M * H * (3 if case["shared"] else 2) + 4.0 * M * E + 8.0 * M * k
    return {"bytes": hit * (3.0 * H * I + scales) + io, "flops": 6.0 * M * k / shards * H * I}


def tolerance(case):
    # bf16 results of fp32 sums; the int8 codes between the two GEMMs may fall to the other side of a rounding
    return {"rel": 1e-2}
