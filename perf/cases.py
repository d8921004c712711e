"""The calls a serving engine makes of this package, as timing cases.

A case is one pass through the public entry points: a fused projection (`VllmFusedFP8LoRA`, `VllmFusedNVFP4LoRA`) on one
batch, the four projections of a decoder layer, or the token sort and segment index of a forward (`KernelMeta`).  Shapes are
those of the benchmark layer (hidden 4096, 12288 intermediate) and of the tensor-parallel shards of the 72B-class layer
(hidden 8192, 29568 intermediate); batches run from one decode token to a prefill of 8192 tokens, adapters are stored as
bf16, FP8 or NVFP4, ranks 16 to 128, with and without the fused neighbours (SiLU * mul before, residual add behind).

Decode-sized batches are captured in a CUDA graph once, as engines do, and a pass is one replay; prefill batches are called.
"""
from __future__ import annotations

import math

import torch

from onebase_b200.kernels.fp8_lora_vllm import VllmFusedFP8LoRA
from onebase_b200.kernels.nvfp4_lora_vllm import VllmFusedNVFP4LoRA
from onebase_b200.metadata import KernelMeta

DEV = "cuda"
MAX_M = 8192              # the engine's most tokens per forward: every layer is built for it, whatever the batch
GRAPH_M = 256             # batches up to this size are replayed from a CUDA graph
SHAPES = {                # name -> (input features, widths of the merged outputs)
    "qkv": (4096, (4096, 1024, 1024)),
    "o": (4096, (4096,)),
    "gate_up": (4096, (12288, 12288)),
    "down": (12288, (4096,)),
    "tp8_qkv": (8192, (1024, 128, 128)),          # one rank of eight of the 72B-class layer
    "tp8_gate_up": (8192, (3696, 3696)),
    "tp8_down": (3696, (8192,)),
    "tp4_gate_up": (8192, (7392, 7392)),
}
LAYER = ("qkv", "o", "gate_up", "down")


def _case(shape, M, batch, base="fp8", adapters="bf16", tenants=32, rank=64, silu=False, residual=False):
    return {"kind": "projection", "shape": shape, "tokens": M, "batch": batch, "base": base, "adapters": adapters,
            "tenants": tenants, "rank": rank, "silu": silu, "residual": residual}


def listed():
    return [
        # the benchmark's step: a decoder layer's four projections, every one of 32 sequences with an adapter of its own choice
        {"name": "decode_layer", "kind": "layer", "tokens": 32, "batch": "decode", "base": "fp8", "adapters": "bf16",
         "tenants": 32, "rank": 64},
        # one user typing: the smallest call, NVFP4 checkpoint
        dict(_case("o", 1, "decode", base="nvfp4", tenants=8), name="decode_one_token"),
        # an odd number of running sequences, adapters kept in FP8 to fit more of them
        dict(_case("qkv", 23, "decode", adapters="fp8"), name="decode_fp8_adapters"),
        # a full decode batch on the NVFP4 checkpoint with NVFP4-stored adapters, the widest projection
        dict(_case("gate_up", 32, "decode", base="nvfp4", adapters="nvfp4"), name="decode_nvfp4_adapters"),
        # chunked prefill: running decodes and a piece of one prompt in the same forward
        dict(_case("gate_up", 200, "mixed"), name="mixed_batch"),
        # prompts of several tenants of rank 16, few adapters loaded, ragged size
        dict(_case("qkv", 777, "prefill", tenants=4, rank=16), name="prefill_rank16"),
        # one rank of a tensor-parallel layer whose slices are no multiple of any tile
        dict(_case("tp8_gate_up", 512, "prefill"), name="prefill_tp_shard"),
        # the down projection with the activation before it and the residual stream behind it
        dict(_case("down", 2048, "prefill", silu=True, residual=True), name="prefill_down_fused"),
        # NVFP4 checkpoint, FP8-stored adapters: the configurations' prefill
        dict(_case("gate_up", 2048, "prefill", base="nvfp4", adapters="fp8"), name="prefill_fp8_adapters"),
        # the same with NVFP4-stored adapters, ragged size
        dict(_case("o", 1111, "prefill", base="nvfp4", adapters="nvfp4"), name="prefill_nvfp4_adapters"),
        # the largest forward of the widest projection
        dict(_case("gate_up", 8192, "prefill"), name="prefill_largest"),
        # what every forward does first: sort the batch's tokens by adapter
        {"name": "batch_index", "kind": "index", "tokens": 8192, "batch": "prefill", "tenants": 32},
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.49)))))))


def draw(rng):
    kind = rng.choice(["projection"] * 10 + ["layer", "index"])
    tenants = rng.choice([1, 3, 4, 8, 16, 32])
    if kind == "index":
        M = _log_int(rng, 1, MAX_M)
        return {"kind": "index", "tokens": M, "batch": rng.choice(["decode", "prefill", "mixed"]), "tenants": tenants}
    rank = rng.choice([16, 32, 64, 64, 128])
    base = rng.choice(["fp8", "nvfp4"])
    adapters = rng.choice(["bf16", "bf16", "fp8", "nvfp4"])
    if kind == "layer":
        M = _log_int(rng, 1, 32)
        return {"kind": "layer", "tokens": M, "batch": "decode", "base": base, "adapters": adapters, "tenants": tenants,
                "rank": rank}
    shape = rng.choice([s for s in SHAPES if base == "fp8" or not s.startswith("tp")])
    batch = rng.choice(["decode", "mixed", "prefill", "prefill"])
    if batch == "decode":
        M = _log_int(rng, 1, 256)
    elif batch == "mixed":
        M = _log_int(rng, 33, 512)
    else:
        M = _log_int(rng, 64, 2048)
    down = shape in ("down", "tp8_down")
    return _case(shape, M, batch, base=base, adapters=adapters, tenants=tenants, rank=rank,
                 silu=down and rng.random() < 0.5, residual=(down or shape == "o") and rng.random() < 0.5)


# ---------------------------------------------------------------------------------------------------------------- inputs
def _zipf_counts(M, tenants):
    share = 1.0 / torch.arange(1, tenants + 1, dtype=torch.float64) ** 1.1
    exact = share / share.sum() * M
    counts = exact.floor().long()
    counts[torch.argsort(exact - counts, descending=True)[: M - int(counts.sum())]] += 1
    return counts


def _slot_ids(case, seed):
    """Adapter slot of every token (-1: none).  decode: a slot per sequence, one in sixteen without; prefill: prompts of
    contiguous tokens whose sizes follow Zipf(1.1) over the tenants; mixed: 32 decoding sequences, then a piece of one prompt
    and the last piece of another."""
    M, L, g = case["tokens"], case["tenants"], torch.Generator().manual_seed(seed)
    if case["batch"] == "prefill":
        return torch.repeat_interleave(torch.randperm(L, generator=g).to(torch.int32), _zipf_counts(M, L)[torch.randperm(L, generator=g)])
    n = M if case["batch"] == "decode" else min(32, M)
    ids = torch.randint(0, L, (n,), generator=g, dtype=torch.int32)
    ids[torch.rand(n, generator=g) < 1.0 / 16] = -1
    a, b = int(torch.randint(0, L, (1,), generator=g)), int(torch.randint(0, L, (1,), generator=g))
    rest = M - n
    return torch.cat([ids, torch.full((rest - rest // 4,), a, dtype=torch.int32), torch.full((rest // 4,), b, dtype=torch.int32)])


def _distinct(case):
    L, M = case["tenants"], case["tokens"]
    if case["batch"] == "prefill":
        return int((_zipf_counts(M, L) > 0).sum())
    n = M if case["batch"] == "decode" else min(32, M)
    return min(L, L * (1.0 - (1.0 - 1.0 / L) ** n) + (2 if M > n else 0))


_E2M1 = (0.0, 0.5, 1.0, 1.5, 2.0, 3.0, 4.0, 6.0)


def _nvfp4(t, gs):
    """vLLM's block recipe: t [..., k], global multiplier gs (broadcastable, fp32) -> (e2m1 codes uint8 [..., k], e4m3 scales
    [..., k/16]); one scale per 16 elements, IEEE reciprocals, ties to even."""
    b = t.float().unflatten(-1, (-1, 16))
    gs = gs.unsqueeze(-1)
    sf = (gs * (b.abs().amax(-1, keepdim=True) * (1.0 / 6.0))).clamp(max=448.0).to(torch.float8_e4m3fn)
    sff = sf.float()
    v = b * torch.where(sff != 0, (sff * gs.reciprocal()).reciprocal(), torch.zeros_like(sff))
    a = v.abs()
    code = torch.zeros(b.shape, dtype=torch.uint8, device=t.device)
    for edge, closed in ((0.25, 0), (0.75, 1), (1.25, 0), (1.75, 1), (2.5, 0), (3.5, 1), (5.0, 0)):
        code += (a >= edge) if closed else (a > edge)
    return (code + (v < 0).to(torch.uint8) * 8).flatten(-2), sf.squeeze(-1)


def _nvfp4_value(codes, sf):
    table = torch.tensor(_E2M1 + tuple(-v for v in _E2M1), dtype=torch.float64, device=codes.device)
    return (table[codes.int()].unflatten(-1, (-1, 16)) * sf.double().unsqueeze(-1)).flatten(-2)


def _tensors(case, shape, g):
    """One projection's inputs, drawn on the device: activations N(0, 1), weights N(0, 0.02), A uniform in +-1/sqrt(K) and B
    N(0, 0.01) in vLLM's stacked layout."""
    K, widths = SHAPES[shape]
    N, M, L, R = sum(widths), case["tokens"], case["tenants"], case["rank"]
    t = {"K": K, "widths": widths}
    w = torch.randn(N, K, device=DEV, generator=g) * 0.02
    if case["base"] == "fp8":
        t["s_w"] = (w.abs().amax() / 448.0).reshape(1)
        t["w_q"] = (w / t["s_w"]).to(torch.float8_e4m3fn)
    else:
        t["w_global"] = float(2688.0 / w.abs().amax())
        parts = [_nvfp4(p, torch.full((1, 1), t["w_global"], device=DEV)) for p in w.split(4096)]
        t["w_codes"], t["w_sf"] = torch.cat([p[0] for p in parts]), torch.cat([p[1] for p in parts])
        t["x_global"] = 2688.0 / 4.8
    del w
    t["a"] = tuple(((torch.rand(L, 1, R, K, device=DEV, generator=g) * 2 - 1) / K ** 0.5).to(torch.bfloat16) for _ in widths)
    t["b"] = tuple((torch.randn(L, 1, n, R, device=DEV, generator=g) * 0.01).to(torch.bfloat16) for n in widths)
    t["x"] = torch.randn(M, 2 * K if case.get("silu") else K, device=DEV, generator=g).to(torch.bfloat16)
    t["residual"] = torch.randn(M, N, device=DEV, generator=g).to(torch.bfloat16) if case.get("residual") else None
    return t


def _inputs(case, seed):
    g = torch.Generator(device=DEV).manual_seed(seed)
    names = LAYER if case["kind"] == "layer" else (case["shape"],)
    for name in names:
        yield _tensors(case, name, g)


def prepare(case, seed):
    """The op objects of the layer (weights and adapter buffers laid out once), the batch, its index and, for decode-sized
    batches, the captured graph.  For the index alone: the mapping and the metadata object."""
    ids = _slot_ids(case, seed).to(DEV)
    meta = KernelMeta.make(case["tenants"], MAX_M, DEV)
    if case["kind"] == "index":
        return {"kind": "index", "meta": meta, "ids": ids}
    meta.prepare_tensors(ids)
    state = {"kind": "calls", "meta": meta.meta_args(case["tokens"]), "calls": [], "graph": None}
    for t in _inputs(case, seed):
        if case["base"] == "fp8":
            op = VllmFusedFP8LoRA(t["w_q"], t["s_w"], t["a"], t["b"], max_m=MAX_M, lora_fp8=case["adapters"] == "fp8",
                                  lora_fp4=case["adapters"] == "nvfp4")
        else:
            pair = t["w_codes"].unflatten(-1, (-1, 2))
            op = VllmFusedNVFP4LoRA(pair[..., 0] | (pair[..., 1] << 4), t["w_sf"], t["w_global"], t["x_global"], t["a"], t["b"],
                                    max_m=MAX_M, lora_fmt=case["adapters"])
        y = torch.empty(case["tokens"], op.N, dtype=torch.bfloat16, device=DEV)
        state["calls"].append((op, t["x"], y, bool(case.get("silu")), t["residual"]))
    if case["tokens"] <= GRAPH_M:
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            _call_all(state)
        torch.cuda.current_stream().wait_stream(side)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            _call_all(state)
        state["graph"] = graph
    return state


def _call_all(state):
    return [op(x, state["meta"], out=y, silu_mul=silu, residual=residual) for op, x, y, silu, residual in state["calls"]]


def run(state):
    if state["kind"] == "index":
        m = state["meta"]
        m.prepare_tensors(state["ids"])
        n = state["ids"].numel()
        return {"tok": m.token_lora_mapping[:n], "srt": m.token_indices_sorted_by_lora_ids[:n], "seg_n": m.num_tokens_per_lora,
                "seg_start": m.lora_token_start_loc, "seg_ids": m.active_lora_ids}
    if state["graph"] is not None:
        state["graph"].replay()
        return [y for _, _, y, _, _ in state["calls"]]
    return _call_all(state)


# ---------------------------------------------------------------------------------------------------------------- work
def work(case):
    M, L = case["tokens"], case["tenants"]
    if case["kind"] == "index":
        return {"bytes": 4 * (3 * M + 3 * L + 4), "flops": 0}
    names = LAYER if case["kind"] == "layer" else (case["shape"],)
    R, d = case["rank"], _distinct(case)
    total, flops = 16 * M, 0.0
    for name in names:
        K, widths = SHAPES[name]
        N, S = sum(widths), len(widths)
        rows_a, rows_b = S * R, N
        if case["adapters"] == "bf16":
            ad = 2.0 * (rows_a * K + rows_b * R)
        elif case["adapters"] == "fp8":
            ad = rows_a * (K + 4.0) + rows_b * (R + 4.0)
        else:
            ad = 0.5625 * (rows_a * K + rows_b * R) + 8.0 * S
        x = M * K * (4 if case.get("silu") else 2)
        y = M * N * (4 if case.get("residual") else 2)
        total += N * K * (1.0 if case["base"] == "fp8" else 0.5625) + d * ad + x + y
        flops += 2.0 * M * (N * K + S * R * K + N * R)
    return {"bytes": total, "flops": flops}


# ---------------------------------------------------------------------------------------------------------------- results
def tolerance(case):
    """Whole numbers for the index.  Projections round y to bf16 once (1.7e-3 in the 2-norm, 4e-3 in the largest value, as
    measured against 64 bits), twice where a residual is added (2.3e-3 and 1.1e-2); the bf16 rounding of the shrink's result and
    of stored adapters' dequantized B adds little to that, as the LoRA term is a small part of y.  Four times these."""
    if case["kind"] == "index":
        return "exact"
    return {"rel": 9e-3, "max": 4.5e-2} if case.get("residual") else {"rel": 7e-3, "max": 1.7e-2}


def _top():
    """448 as a tensor: torch divides a device tensor by a Python number through its reciprocal, which is not the scale's
    IEEE division."""
    return torch.tensor(448.0, device=DEV)


def _exact_projection(case, ids, t):
    K, widths = t["K"], t["widths"]
    x = t["x"]
    if case.get("silu"):
        x = torch.nn.functional.silu(x[:, :K].float()).to(torch.bfloat16) * x[:, K:]
    if case["base"] == "fp8":
        sx = (x.float().abs().amax(1, keepdim=True) / _top()).clamp_min(1.0 / (448.0 * 512.0))
        xq = (x.float() / sx).clamp(-448.0, 448.0).to(torch.float8_e4m3fn).double()
        y = (xq @ t["w_q"].double().t()) * sx.double() * t["s_w"].double()
    else:
        gs = torch.full((1, 1), t["x_global"], device=DEV)
        xv = _nvfp4_value(*_nvfp4(x, gs))
        wv = torch.cat([_nvfp4_value(c, s) for c, s in zip(t["w_codes"].split(4096), t["w_sf"].split(4096))])
        y = (xv @ wv.t()) / (t["x_global"] * t["w_global"])
    x64 = x.double()
    for l in torch.unique(ids).tolist():
        if l < 0:
            continue
        rows, off = torch.nonzero(ids == l).flatten(), 0
        for a, b in zip(t["a"], t["b"]):
            n = b.shape[2]
            h = x64[rows] @ _stored_value(case, a[l, 0]).t()
            y[rows, off:off + n] += h @ _stored_value(case, b[l, 0]).t()
            off += n
    if t["residual"] is not None:
        y += t["residual"].double()
    return y


def _stored_value(case, m):
    """An adapter matrix [rows, cols] as its storage format holds it."""
    if case["adapters"] == "bf16":
        return m.double()
    f = m.float()
    if case["adapters"] == "fp8":
        scale = (f.abs().amax(-1, keepdim=True) / _top()).clamp_min(1e-12)
        return (f / scale).clamp(-448.0, 448.0).to(torch.float8_e4m3fn).double() * scale.double()
    gs = (f.abs().amax().clamp_min(1e-12).reciprocal() * 2688.0).reshape(1, 1)
    return _nvfp4_value(*_nvfp4(f, gs)) * gs.reciprocal().double()


def exact(case, seed):
    ids = _slot_ids(case, seed).to(DEV)
    if case["kind"] != "index":
        return [_exact_projection(case, ids, t) for t in _inputs(case, seed)]
    M, L = case["tokens"], case["tenants"]
    uniq, counts = torch.unique(ids, return_counts=True)
    out = {"tok": ids, "srt": torch.sort(ids, stable=True).indices.int(), "seg_n": torch.zeros(L + 1, dtype=torch.int32, device=DEV),
           "seg_start": torch.zeros(L + 2, dtype=torch.int32, device=DEV),
           "seg_ids": torch.full((L + 1,), -1, dtype=torch.int32, device=DEV)}
    if bool((ids == -1).all()):                # an all-base batch leaves the index as it was; a new one is empty
        out["tok"], out["srt"] = torch.zeros_like(ids), torch.zeros_like(ids)
        return out
    n = uniq.numel()
    out["seg_n"][:n], out["seg_ids"][:n] = counts.int(), uniq.int()
    out["seg_start"][1:n + 1] = torch.cumsum(counts, 0).int()
    return out
