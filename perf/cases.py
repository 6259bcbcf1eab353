"""Workloads of the decode path with sizes of real use, for timing and for comparing two builds.

Every pass goes through the package's public entry points: ``fast_kernels.ops`` (the W4A16 linear
layer, weight preparation, paged-KV attention and its planner) and, for the fused decoder layer, the
C ABI that ``fast_kernels.capi`` binds. A case is a dict of plain values; its ``kind`` is one of

  linear     ``arc_w4a16_forward``: one quantised layer over a batch of rows
  decoder    the four linear layers of decoder blocks with their fused norm / residual / SiLU options
  attention  ``clustered_page_decode``: one decode token per request over a paged KV cache
  prefix     ``prefix_union_decode``: the same where groups of requests share their first pages
  weights    ``pack_arc_w4a16_packets`` and ``dequant_arc_w4a16_packets``: a layer is loaded, and read back

``listed()`` gives the fixed cases, ``draw(rng)`` another one from the same ranges.
"""

from __future__ import annotations

import ctypes
import dataclasses
import math
import os
import sys

import torch

# the package of the tree that is the working folder, which may be another one than this file's
sys.path.insert(0, os.path.join(os.getcwd(), "fast-kernels_b200", "src"))

from fast_kernels import capi, ops  # noqa: E402

DTYPES = {"fp16": torch.float16, "bf16": torch.bfloat16}
CODES = {"fp16": capi.DTYPE_F16, "bf16": capi.DTYPE_BF16}
ROPE_THETA = 10000.0
NORM_EPS = 1e-5

# Bounds of the ranges: rows of a linear layer (one token of one request up to the tokens of a large
# decode batch or of a piece of a prompt), weights of a layer (up to a 128k-row LM head), and
# multiply-adds of a call.
MAX_ROWS = 256
MAX_WEIGHTS = 128256 * 4096
MAX_MACS = 256 * 28672 * 8192
# KV bytes of one layer and step: 32 requests x 4096 tokens x 8 heads x 128 dims in bf16.
MAX_KV_BYTES = 32 * 4096 * 8 * 128 * 2 * 2


def listed() -> list[dict]:
    return [
        # The smallest call: one 4096 x 4096 projection, one row. What counts is latency.
        dict(name="linear_4096_m1", kind="linear", dtype="fp16", group=128, m=1, n=4096, k=4096, zeros="fixed"),
        # A few rows (parallel samples of one request) on a 13B MLP layer with small groups.
        dict(name="linear_13b_g32_m3", kind="linear", dtype="fp16", group=32, m=3, n=13824, k=5120, zeros="any"),
        # A small decode batch on a 70B-style MLP up projection.
        dict(name="linear_70b_m8", kind="linear", dtype="bf16", group=128, m=8, n=28672, k=8192, zeros="any"),
        # The serving batch of the attention cases on the 8B gate/up layer.
        dict(name="linear_8b_m32", kind="linear", dtype="bf16", group=128, m=32, n=28672, k=4096, zeros="fixed"),
        # A large decode batch, or a piece of a prompt, on the 70B-style layer: the most arithmetic.
        dict(name="linear_70b_m256", kind="linear", dtype="bf16", group=128, m=256, n=28672, k=8192, zeros="any"),
        # The LM head for one token: the largest single layer.
        dict(name="linear_lm_head_m1", kind="linear", dtype="bf16", group=128, m=1, n=128256, k=4096, zeros="fixed"),
        # One token through four decoder blocks of the 8B model, fused callers, weights from HBM.
        dict(name="decoder_8b_m1", kind="decoder", dtype="bf16", group=128, m=1, hidden=4096, qkv=6144, inter=14336,
             blocks=4),
        # Short contexts, small heads: a call of a few microseconds.
        dict(name="attention_short_d64", kind="attention", layout="bf16_kv", rotated=False, requests=8, shortest=480,
             longest=512, q_heads=16, kv_heads=8, head_dim=64, page=32, layers=1, plan="kept"),
        # Two long contexts, grouped by eight, quantised pages whose keys are turned in the kernel.
        dict(name="attention_long_int8", kind="attention", layout="int8_kv", rotated=False, requests=2, shortest=4070,
             longest=4096, q_heads=32, kv_heads=4, head_dim=128, page=32, layers=1, plan="kept"),
        # A serving step: 32 requests of mixed length, planned once for the step, two layers of it.
        dict(name="attention_serving_step", kind="attention", layout="bf16_kv", rotated=True, requests=32, shortest=1024,
             longest=4096, q_heads=32, kv_heads=8, head_dim=128, page=16, layers=2, plan="step"),
        # Requests that share a system prompt, e4m3 pages with turned keys.
        dict(name="prefix_fp8", kind="prefix", layout="fp8_kv", rotated=True, requests=8, shortest=1200, longest=2048,
             q_heads=32, kv_heads=8, head_dim=128, page=16, shared_pages=8, sharers=4),
        # Loading the 8B gate/up layer, and its dense form for a caller that wants one.
        dict(name="weights_8b_gate_up", kind="weights", dtype="bf16", group=128, n=28672, k=4096),
    ]


# ---- drawn cases -----------------------------------------------------------------------------------


def _log(rng, low: float, high: float) -> float:
    return math.exp(rng.uniform(math.log(low), math.log(high)))


def _multiple(rng, low: int, high: int, step: int) -> int:
    return max(low, min(high, round(_log(rng, low, high) / step) * step))


def _draw_layer(rng, group: int) -> tuple[int, int]:
    while True:
        n, k = _multiple(rng, 512, 128256, 128), _multiple(rng, 1024, 28672, group)
        if n * k <= MAX_WEIGHTS:
            return n, k


def _draw_kv(rng, layout: str, limit: int) -> dict:
    while True:
        kv_heads, share = rng.choice((1, 2, 4, 8)), rng.choice((1, 2, 3, 4, 6, 8, 12, 32))
        dim, page = rng.choice((64, 128)), rng.choice((16, 32))
        requests, longest = round(_log(rng, 1, 64)), round(_log(rng, 64, 16384))
        element = 2 if layout == "bf16_kv" else 1
        if kv_heads * share <= 64 and requests * longest * kv_heads * dim * 2 * element <= limit:
            return dict(requests=requests, shortest=max(1, round(longest * rng.uniform(0.1, 1.0))), longest=longest,
                        q_heads=kv_heads * share, kv_heads=kv_heads, head_dim=dim, page=page)


def draw(rng) -> dict:
    kind = rng.choice(("linear", "linear", "linear", "decoder", "attention", "attention", "prefix", "weights"))
    dtype, group = rng.choice(("bf16", "fp16")), rng.choice((32, 64, 128))
    if kind == "linear":
        while True:
            (n, k), m = _draw_layer(rng, group), round(_log(rng, 1, MAX_ROWS))
            if m * n * k <= MAX_MACS:
                return dict(kind=kind, dtype=dtype, group=group, m=m, n=n, k=k, zeros=rng.choice(("fixed", "any")))
    if kind == "decoder":
        m, hidden = rng.randint(1, 4), _multiple(rng, 1024, 4096, 128)
        inter = _multiple(rng, 2 * hidden, min(4 * hidden, 14336), 128)
        qkv = hidden + 2 * rng.choice((128, 256, 512, 1024))
        return dict(kind=kind, dtype=dtype, group=group, m=m, hidden=hidden, qkv=qkv, inter=inter, blocks=rng.randint(1, 4))
    layout = rng.choice(("bf16_kv", "fp8_kv", "int8_kv"))
    if kind == "attention":
        plan = rng.choice(("kept", "step"))
        layers = rng.randint(1, 2) if plan == "step" else 1
        return dict(kind=kind, layout=layout, rotated=rng.random() < 0.5, layers=layers, plan=plan,
                    **_draw_kv(rng, layout, MAX_KV_BYTES))
    if kind == "prefix":
        shape = _draw_kv(rng, layout, MAX_KV_BYTES // 16)
        shape["requests"] = max(2, shape["requests"])
        shared = rng.randint(1, 8)
        shape["shortest"] = max(shape["shortest"], shared * shape["page"] + 1)
        shape["longest"] = max(shape["longest"], shape["shortest"])
        return dict(kind=kind, layout=layout, rotated=True, shared_pages=shared, sharers=rng.randint(2, 4), **shape)
    while True:
        n, k = _draw_layer(rng, group)
        if n * k <= 28672 * 4096:
            return dict(kind=kind, dtype=dtype, group=group, n=n, k=k)


# ---- inputs ----------------------------------------------------------------------------------------


def _quantised(gen, n: int, k: int, group: int, dtype, zeros: str) -> tuple:
    """(nibbles, scales, offsets) as a loader has them: uniform int4, offset = -(scale * zero point)."""
    q = torch.randint(0, 256, (n, k // 2), generator=gen, device="cuda", dtype=torch.uint8)
    alpha = (0.005 + 0.015 * torch.rand((n, k // group), generator=gen, device="cuda")).to(dtype)
    if zeros == "fixed":
        return q, alpha, -(alpha * 8)
    points = torch.randint(0, 16, (n, k // group), generator=gen, device="cuda").to(dtype)
    return q, alpha, -(alpha * points)


def _packed(gen, n: int, k: int, group: int, dtype, zeros: str = "fixed"):
    return ops.pack_arc_w4a16_packets(*_quantised(gen, n, k, group, dtype, zeros), group_size=group)


def _rows(gen, m: int, width: int, dtype):
    return torch.randn((m, width), generator=gen, device="cuda").to(dtype)


def _lengths(case: dict) -> list[int]:
    """The requests' lengths: even steps from the shortest to the longest, whatever the seed."""
    count, low, high = case["requests"], case["shortest"], case["longest"]
    return [high - (high - low) * i // max(1, count - 1) for i in range(count)]


def _kv_cache(case: dict, gen, lens):
    """A cache as the package's own builders make it: pages anywhere in the pool, no two neighbours by design."""
    shape = (case["requests"], case["kv_heads"], case["longest"], case["head_dim"])
    build = {"bf16_kv": ops.pack_paged_kv_bf16, "fp8_kv": ops.quantize_paged_kv_fp8, "int8_kv": ops.quantize_paged_kv_int8}
    keys, values = (torch.randn(shape, generator=gen, device="cuda", dtype=torch.bfloat16) for _ in range(2))
    return build[case["layout"]](keys, values, lens, page_size=case["page"], seed=gen.initial_seed() % (1 << 31),
                                 key_rope_theta=ROPE_THETA if case["rotated"] else None)


def _plan_arguments(case: dict, cache) -> dict:
    return dict(page_table=cache.page_table, seq_lens=cache.seq_lens, num_q_heads=case["q_heads"],
                num_kv_heads=case["kv_heads"], head_dim=case["head_dim"], page_size=case["page"],
                kv_layout=case["layout"])


def _prepare_decoder(case: dict, gen, dtype) -> dict:
    """Weights, buffers and the argument structs of the calls, which such a program fills in once."""
    m, hidden, qkv, inter, group = (case[key] for key in ("m", "hidden", "qkv", "inter", "group"))
    lib, stride = capi.load_library(), capi.packet_stride_bytes(group)
    need = max(int(lib.fk_w4a16_workspace_bytes(m, n, k, group))
               for n, k in ((qkv, hidden), (hidden, hidden), (2 * inter, hidden), (hidden, inter)))
    workspace = torch.zeros(need, dtype=torch.uint8, device="cuda")
    keep, calls, outputs = [workspace], [], []

    def call(activations, n, k, output, residual=None, norm=None, epilogue=capi.EPILOGUE_NONE) -> None:
        packets = _packed(gen, n, k, group, dtype)
        a = capi.GemvArgs()
        a.activations, a.packets, a.output = activations.data_ptr(), packets.data_ptr(), output.data_ptr()
        a.workspace, a.workspace_bytes = workspace.data_ptr(), workspace.numel()
        a.batch, a.n, a.k, a.group_size, a.packet_stride_bytes, a.dtype = m, n, k, group, stride, CODES[case["dtype"]]
        a.residual = 0 if residual is None else residual.data_ptr()
        if norm is not None:
            a.norm_weight, a.norm_eps = norm.data_ptr(), NORM_EPS
        a.epilogue = epilogue
        a.stream = int(torch.cuda.current_stream().cuda_stream)
        keep.extend((activations, packets, output, residual, norm))
        calls.append(a)

    def empty(width: int):
        return torch.empty((m, width), dtype=dtype, device="cuda")

    h = _rows(gen, m, hidden, dtype)
    for _ in range(case["blocks"]):
        norms = [(1.0 + 0.05 * torch.randn(hidden, generator=gen, device="cuda")).to(dtype) for _ in range(2)]
        attended = (0.5 * torch.randn((m, hidden), generator=gen, device="cuda")).to(dtype)
        projected, middle, gated, after = empty(qkv), empty(hidden), empty(inter), empty(hidden)
        call(h, qkv, hidden, projected, norm=norms[0])
        call(attended, hidden, hidden, middle, residual=h)
        call(middle, 2 * inter, hidden, gated, norm=norms[1], epilogue=capi.EPILOGUE_SILU_MUL)
        call(gated, hidden, inter, after, residual=middle)
        outputs += [projected, gated, after]
        h = after
    return dict(kind="decoder", lib=lib, calls=calls, outputs=outputs, keep=keep)


def prepare(case: dict, seed: int) -> dict:
    kind = case["kind"]
    gen = torch.Generator(device="cuda").manual_seed(seed)
    if kind == "linear":
        dtype = DTYPES[case["dtype"]]
        packets = _packed(gen, case["n"], case["k"], case["group"], dtype, case["zeros"])
        return dict(case=case, kind=kind, packets=packets, activations=_rows(gen, case["m"], case["k"], dtype))
    if kind == "decoder":
        return _prepare_decoder(case, gen, DTYPES[case["dtype"]])
    if kind == "weights":
        return dict(case=case, kind=kind,
                    layer=_quantised(gen, case["n"], case["k"], case["group"], DTYPES[case["dtype"]], "any"))
    lens = torch.tensor(_lengths(case), dtype=torch.int32)[torch.randperm(case["requests"],
                                                                         generator=torch.Generator().manual_seed(seed))]
    caches = [_kv_cache(case, gen, lens) for _ in range(case.get("layers", 1))]
    queries = [torch.randn((case["requests"], case["q_heads"], case["head_dim"]), generator=gen, device="cuda").to(torch.bfloat16)
               for _ in caches]
    state = dict(case=case, kind=kind, caches=caches, queries=queries)
    # the layers of a model share the page table; each has pages of its own
    caches[1:] = [dataclasses.replace(c, page_table=caches[0].page_table) for c in caches[1:]]
    if kind == "prefix":
        table = caches[0].page_table.clone()
        for first in range(0, case["requests"], case["sharers"]):
            table[first : first + case["sharers"], : case["shared_pages"]] = table[first, : case["shared_pages"]]
        caches[0] = dataclasses.replace(caches[0], page_table=table)
        state["plan"] = ops.plan_prefix_union_decode(**_plan_arguments(case, caches[0]), keys_are_rotated=True, use_cache=False)
    elif case["plan"] == "kept":
        state["plan"] = ops.plan_clustered_page_decode(**_plan_arguments(case, caches[0]), use_cache=False)
    else:
        state["plan"] = None
    return state


# ---- one pass --------------------------------------------------------------------------------------


def run(state: dict):
    kind = state["kind"]
    if kind == "decoder":
        call = state["lib"].fk_w4a16_gemv_ex
        for arguments in state["calls"]:
            capi.check(call(ctypes.byref(arguments)))
        return state["outputs"]
    case = state["case"]
    if kind == "linear":
        return ops.arc_w4a16_forward(state["activations"], state["packets"], n=case["n"], k=case["k"],
                                     group_size=case["group"])
    if kind == "weights":
        packets = ops.pack_arc_w4a16_packets(*state["layer"], group_size=case["group"])
        dense = ops.dequant_arc_w4a16_packets(packets, n=case["n"], k=case["k"], group_size=case["group"],
                                              dtype=DTYPES[case["dtype"]])
        return packets, dense
    plan = state["plan"]
    if kind == "prefix":
        return ops.prefix_union_decode(state["queries"][0], state["caches"][0], plan=plan, rope_theta=ROPE_THETA)
    if plan is None:
        # every step's lengths are new, so a step's plan is never one that was made before
        plan = ops.plan_clustered_page_decode(**_plan_arguments(case, state["caches"][0]), use_cache=False)
    return [ops.clustered_page_decode(query, cache, plan=plan, rope_theta=ROPE_THETA)
            for query, cache in zip(state["queries"], state["caches"])]


# ---- what a pass cannot do without -----------------------------------------------------------------


def _layer_bytes(n: int, k: int, group: int) -> int:
    return n * k // 2 + 4 * n * (k // group)


def work(case: dict) -> dict:
    kind = case["kind"]
    if kind == "linear":
        m, n, k = case["m"], case["n"], case["k"]
        return dict(bytes=_layer_bytes(n, k, case["group"]) + 2 * m * (n + k), flops=2 * m * n * k)
    if kind == "decoder":
        m, hidden, qkv, inter = case["m"], case["hidden"], case["qkv"], case["inter"]
        layers = ((qkv, hidden), (hidden, hidden), (2 * inter, hidden), (hidden, inter))
        weights = sum(_layer_bytes(n, k, case["group"]) for n, k in layers)
        # a block reads its input, the attention's result and two norms, and writes qkv, gated and hidden rows
        rows = 2 * m * (2 * hidden + qkv + inter + hidden) + 4 * hidden
        return dict(bytes=case["blocks"] * (weights + rows), flops=case["blocks"] * sum(2 * m * n * k for n, k in layers))
    if kind == "weights":
        layer = _layer_bytes(case["n"], case["k"], case["group"])
        return dict(bytes=3 * layer + 2 * case["n"] * case["k"], flops=2 * case["n"] * case["k"])
    lens, page, dim = _lengths(case), case["page"], case["head_dim"]
    tokens, pages = sum(lens), sum(-(-length // page) for length in lens)
    flops = 4 * tokens * case["q_heads"] * dim
    if kind == "prefix":  # the pages that requests share are read once
        groups = -(-case["requests"] // case["sharers"])
        spared = (case["requests"] - groups) * case["shared_pages"]
        tokens, pages = tokens - spared * page, pages - spared
    element = 2 if case["layout"] == "bf16_kv" else 1
    kv = tokens * case["kv_heads"] * dim * 2 * element
    if element == 1:
        kv += (tokens + pages) * case["kv_heads"] * (dim // 64) * 4
    layers = case.get("layers", 1)
    return dict(bytes=layers * (kv + 4 * case["requests"] * case["q_heads"] * dim), flops=layers * flops)


def tolerance(case: dict):
    kind = case["kind"]
    if kind == "weights":  # bytes moved about, and one rounding that is defined exactly
        return "exact"
    if kind == "linear" and case["dtype"] == "fp16":  # one rounding to fp16 behind a 32-bit sum
        return {"rel": 1e-3}
    if kind == "decoder" and case["dtype"] == "fp16":  # several such roundings in a row
        return {"rel": 4e-3}
    return {"rel": 1e-2}
