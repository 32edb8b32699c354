"""Workloads of the MoDA operators: what a model that uses this library has it do, over the range of
sizes, directions, types and options that are in use.

A case is one call (or one training step, or one stack of layers) through the public operators:

  op      "moda" (parallel_moda), "chunk" (parallel_moda_chunk_visible), "fda" (parallel_fda), or
          "stack" (a stack of layers over a DepthKVCache)
  causal  sequence keys up to the query's own position, or all of them ("moda" and "stack")
  train   forward and backward through autograd, or the forward alone (inference)
  B, T, H, G, D   batch, positions, KV heads, query heads of a KV head, head dim
  L       depth layers that the call sees ("stack": layers of the stack; layer i sees i earlier ones)
  dtype   "bfloat16" or "float16"
"""
import math

import torch

import moda_b200 as M

DTYPES = {"bfloat16": torch.bfloat16, "float16": torch.float16}


def _case(op, causal, train, B, T, H, G, D, L, dtype="bfloat16", **more):
    return dict(more, op=op, causal=causal, train=train, B=B, T=T, H=H, G=G, D=D, L=L, dtype=dtype)


def listed():
    return [
        # the smallest call of the operator's own test configurations: what it costs to call it at all
        _case("moda", True, False, 1, 256, 4, 1, 64, 4, name="tiny_forward"),
        # a debugging-size training step in fp16: forward and backward through autograd
        _case("moda", True, True, 2, 192, 4, 2, 64, 8, "float16", name="small_train"),
        # prompt processing of a grouped-query language model, own-position depth
        _case("moda", True, False, 2, 4096, 4, 4, 128, 24, name="prefill_causal"),
        # prompt processing with chunk-visible depth, one long prompt
        _case("chunk", True, False, 1, 8192, 8, 4, 128, 32, name="prefill_chunk_visible"),
        # long-context training step, chunk-visible depth: the headline workload
        _case("chunk", True, True, 1, 65536, 8, 4, 128, 32, name="long_train_chunk_visible"),
        # long-context training step, own-position depth, narrow heads: the published shape
        _case("moda", True, True, 1, 65536, 8, 8, 64, 64, name="long_train_causal"),
        # training step on sequences that fill no tile: odd length, odd head and layer counts
        _case("moda", True, True, 3, 1531, 5, 2, 128, 7, "float16", name="ragged_train"),
        # depth-only attention of a large training step
        _case("fda", True, True, 8, 8192, 16, 1, 128, 32, name="depth_only_train"),
        # depth-only attention with grouped queries, odd length
        _case("fda", True, True, 2, 4093, 4, 4, 128, 24, name="depth_only_train_gqa"),
        # one attention layer of a vision transformer at its training batch
        _case("moda", False, True, 256, 197, 6, 1, 64, 11, name="vision_train"),
        # all attention layers of that vision transformer over the in-place depth cache
        _case("stack", False, True, 64, 197, 6, 1, 64, 12, name="vision_stack_train"),
        # all attention layers of a small grouped-query language model over the in-place depth cache
        _case("stack", True, True, 2, 2048, 4, 4, 128, 12, name="language_stack_train"),
    ]


# A drawn case does less work than the largest listed ones; a stack is up to 16 calls of all sizes.
MOST_FLOPS = {"moda": 60e12, "chunk": 60e12, "fda": 60e12, "stack": 12e12}
MOST_BYTES = 20e9


def _spread(rng, lo, hi):
    """A whole number from lo to hi, spread over the logarithm."""
    return min(hi, max(lo, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def draw(rng):
    while True:
        op = rng.choice(["moda", "moda", "chunk", "fda", "stack"])
        causal = rng.random() < 0.7 if op in ("moda", "stack") else True
        train = True if op == "stack" else rng.random() < 0.6
        if op == "stack":
            L = rng.randint(2, 16)
        elif op == "fda":
            L = rng.randint(2, 64)       # with one depth row the softmax is constant and has no gradient
        else:
            L = rng.randint(0, 64)
        T = _spread(rng, 32, 65536) if causal else _spread(rng, 32, 4096)
        case = _case(op, causal, train, _spread(rng, 1, 256), T, rng.randint(1, 16),
                     rng.choice([1, 2, 4, 8]), rng.choice([64, 128]), L,
                     rng.choice(["bfloat16", "bfloat16", "float16"]))
        w = work(case)
        if w["flops"] <= MOST_FLOPS[op] and w["bytes"] <= MOST_BYTES:
            return case


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    dtype = DTYPES[case["dtype"]]
    B, T, H, G, D, L = (case[x] for x in "BTHGDL")

    def mk(rows, leaf=True):
        x = torch.randn(B, rows, H, D, generator=gen, device="cuda", dtype=dtype)
        return x.requires_grad_(case["train"] and leaf)

    state = {"case": case}
    if case["op"] == "stack":
        state["layers"] = [(mk(T * G), mk(T), mk(T)) for _ in range(L)]
        state["dout"] = [mk(T * G, leaf=False) for _ in range(L)]
        state["cache"] = M.DepthKVCache(B, T, L - 1, H, D, dtype, "cuda")
        return state
    state["q"] = mk(T * G)
    if case["op"] != "fda":
        state["k"], state["v"] = mk(T), mk(T)
    if L > 0:
        state["depth_k"], state["depth_v"] = mk(T * L), mk(T * L)
    if case["train"]:
        state["dout"] = mk(T * G, leaf=False)
    return state


def _call(s):
    case, kd, vd = s["case"], s.get("depth_k"), s.get("depth_v")
    G = case["G"]
    if case["op"] == "fda":
        return M.parallel_fda(s["q"], cached_k=kd, cached_v=vd, moda_group_num=G, need_lse=True)
    if case["op"] == "chunk":
        return M.parallel_moda_chunk_visible(s["q"], s["k"], s["v"], cached_k=kd, cached_v=vd,
                                             moda_group_num=G, need_lse=True)
    return M.parallel_moda(s["q"], s["k"], s["v"], cached_k=kd, cached_v=vd, moda_group_num=G,
                           is_causal=case["causal"], need_lse=True)


def run(state):
    case = state["case"]
    if case["op"] == "stack":
        cache = state["cache"]
        cache.reset()
        outs = []
        for i, (q, k, v) in enumerate(state["layers"]):
            outs.append(cache.attend(q, k, v, moda_group_num=case["G"], is_causal=case["causal"]))
            if i + 1 < case["L"]:
                cache.append(k, v)
        leaves = [x for layer in state["layers"] for x in layer]
        grads = torch.autograd.grad(outs, leaves, state["dout"])
        return [o.detach() for o in outs] + list(grads)
    if not case["train"]:
        with torch.no_grad():
            return _call(state)
    o, lse = _call(state)
    leaves = [state[x] for x in ("q", "k", "v", "depth_k", "depth_v") if x in state]
    return [o.detach(), lse] + list(torch.autograd.grad(o, leaves, state["dout"]))


def _pairs(case, L):
    """(query row, key) pairs that the visibility rule lets through, over all heads."""
    B, T, H, G = (case[x] for x in "BTHG")
    if case["op"] == "fda":
        seq = 0
    else:
        seq = T * (T + 1) // 2 if case["causal"] else T * T
    if case["op"] == "chunk":           # a query sees the depth rows of its 64-row chunk up to its own
        C = M.CHUNK_VISIBLE_QUERY_ROWS // G
        full, rest = divmod(T, C)
        depth = L * (full * (C * (C + 1) // 2) + rest * (rest + 1) // 2)
    else:
        depth = L * T
    return B * H * G * (seq + depth)


def work(case):
    """Forward: q, k, v, depth K/V read, o and lse written.  Backward: those and dout read, the five
    gradients written.  4 D flops of a pair forward, 10 D backward (S, P V; S, dP, dQ, dK, dV).  In a
    stack every layer reads the depth rows of the layers before it, in each direction."""
    B, T, H, G, D, L = (case[x] for x in "BTHGDL")
    row = B * T * H * D * 2
    lse = B * T * G * H * 4
    q = G * row
    kv = 0 if case["op"] == "fda" else 2 * row
    if case["op"] == "stack":
        flops = sum(14 * D * _pairs(case, i) for i in range(L))
        depth = sum(2 * i * row for i in range(L))
        return {"bytes": L * (6 * q + 3 * kv + 2 * lse) + 2 * depth, "flops": flops}
    pairs, depth = _pairs(case, L), 2 * L * row
    if not case["train"]:
        return {"bytes": 2 * q + kv + depth + lse, "flops": 4 * D * pairs}
    return {"bytes": 6 * q + 3 * kv + 3 * depth + 2 * lse, "flops": 14 * D * pairs}


def tolerance(case):
    """Probabilities, score gradients and results are rounded to the data type between and after the
    matmuls, with fp32 accumulation: a few roundings of 2^-9 (bf16) or 2^-12 (fp16) relative."""
    return {"rel": 1e-2} if case["dtype"] == "bfloat16" else {"rel": 2e-3}
