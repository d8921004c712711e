"""Stored adapters (FP8 and NVFP4 codes) in prefill: the tensor-core shrink that turns A's codes into operand tiles and the
CTA-pair GEMM that does the same with B's, over both bases, ranks of one to four expand chunks and below one, slices that end
inside a tile, K that ends inside a k step, tenant groups and several accumulator passes -- h against the product with the
dequantized A, y within 2e-2 * ||y||inf of the oracle on the dequantized adapters."""
from __future__ import annotations

import pytest
import torch

from helpers import build_fp8_op, build_nvfp4_op, device_meta, make_index, max_err_ratio, stored_adapters
from onebase_b200.kernels import fp8_lora_vllm
from oracle import configs, fp8 as ofp8, nvfp4 as on4, segments as oseg

pytestmark = pytest.mark.gpu
TOL = 2e-2


# (the last two: on an FP8 base 512-feature tiles, several per CTA pair, whole and ragged slices)
CASES = [(512, (264, 120, 1000), 16, 5, 129), (1024, (512, 8), 64, 40, 300), (528, (776,), 32, 3, 517), (512, (640, 256), 128, 7, 700),
         (256, (384,), 256, 3, 150), (2048, (256, 512), 64, 9, 1000),
         (512, (20480,), 64, 7, 1037), (256, (16392, 4096), 32, 30, 900)]


@pytest.mark.parametrize("fmt", ["fp8", "nvfp4"])
@pytest.mark.parametrize("base", ["fp8", "nvfp4"])
@pytest.mark.parametrize("K,widths,R,L,M", CASES)
def test_stored_adapters_prefill(base, fmt, K, widths, R, L, M):
    if base == "nvfp4" and K % 256:
        K = 768                                               # (an NVFP4 base takes the large tiles in whole 256-element k-blocks)
    d = configs.draw(K, widths, R, L, M, seed=K + M + R, ids_low=-1, w_std=0.05, b_std=0.05)
    d["ids"] = configs.zipf_request_ids(M, L, seed=M, mean_len=30)
    d["ids"][60:75] = -1
    if base == "fp8":
        d = configs.with_fp8_base(d)
        op = build_fp8_op(d, max_m=M, lora_fp8=fmt == "fp8", lora_fp4=fmt == "nvfp4")
    else:
        d = configs.with_nvfp4_base(d)
        op = build_nvfp4_op(d, max_m=M, lora_fmt=fmt)
    big = {"prefill": 1}                                      # (the rule keeps some of these on the smaller tiles)
    assert op.resolved_tile(M, big)["prefill"] == 1
    idx = make_index(d["ids"], L, M)
    meta, x = device_meta(idx, M), d["x"].cuda()
    y = op(x, meta, cfg=big)
    y2 = op(x, meta, out=torch.full_like(y, 7.0), cfg=big)
    torch.cuda.synchronize()
    assert op.scratch.status()[0] == 0, op.scratch.status()[:8]
    A, B = stored_adapters(op, fmt)
    if base == "fp8":
        ref = ofp8.fused_projection(d["x"], d["ids"], d["w_q"], d["s_w"], A, B, widths)
    else:
        ref = on4.fused_projection(d["x"], d["ids"], d["w_q4"], d["w_sf"], d["w_global"], d["x_global"], A, B, widths)
    assert max_err_ratio(y, ref) <= TOL and torch.equal(y, y2)
    # the finished h on the smaller tiles: bf16 of an fp32 sum, so within one and a half bf16 spacings (2^-7 |h| at most) of the
    # fp32 product, and 2e-5 of the largest for the sums' order
    y3 = op(x, meta, cfg={"prefill": 1, "tn": 64})
    torch.cuda.synchronize()
    assert op.scratch.status()[0] == 0 and max_err_ratio(y3, ref) <= TOL
    rows, _ = oseg.resolve_positions(M, *idx.args(M))
    has = d["ids"][rows] >= 0
    hb = op.scratch.hb(len(widths), R).float().cpu()[:, :M].permute(1, 0, 2)[has]
    xs, ids = d["x"].float()[rows][has], d["ids"][rows][has].long()
    want = torch.stack([A[l] @ v for v, l in zip(xs, ids)]).view(-1, len(widths), R)
    bound = 1.5 * 2.0 ** -7 * want.abs() + 2e-5 * float(want.abs().max())
    assert bool(((hb - want).abs() <= bound).all())


@pytest.mark.parametrize("fmt", ["bf16", "fp8"])
def test_batches_beyond_the_shrinks_counters(fmt, monkeypatch):
    """More (tile, tenant group, slice) work items than the tensor-core shrink has arrival counters: the warp-level form serves
    the call."""
    monkeypatch.setattr(fp8_lora_vllm, "_SCRATCH", {})        # (a workspace of its own: the shared one would stay this large)
    M, K, widths, L = 131_200, 64, (16, 16, 16, 16), 4
    d = configs.with_fp8_base(configs.draw(K, widths, 16, L, M, seed=1, ids_low=-1, w_std=0.05, b_std=0.05))
    op = build_fp8_op(d, max_m=M, lora_fp8=fmt == "fp8")
    assert op.resolved_tile(M)["prefill"] == 2 and op.resolved_tile(131_072)["prefill"] == 1
    y = op(d["x"].cuda(), device_meta(make_index(d["ids"], L, M), M))
    torch.cuda.synchronize()
    assert op.scratch.status()[0] == 0
    A, B = stored_adapters(op, fmt)
    ref = ofp8.fused_projection(d["x"], torch.full_like(d["ids"], -1), d["w_q"], d["s_w"], A, B, widths)
    ref += ofp8.lora_term(d["x"], d["ids"], A, B, widths, grouped=True)
    assert max_err_ratio(y, ref) <= TOL


@pytest.mark.parametrize("base,fmt,K,N,L,R,M,large", [
    ("nvfp4", "fp8", 4096, 4096, 4, 64, 256, False), ("nvfp4", "fp8", 4096, 4096, 5, 64, 256, True),
    ("nvfp4", "fp8", 4096, 4096, 4, 64, 257, True), ("nvfp4", "fp8", 4352, 4096, 1, 16, 200, True),
    ("nvfp4", "nvfp4", 4096, 4096, 8, 128, 129, False), ("nvfp4", "nvfp4", 4096, 4096, 9, 128, 129, True),
    ("nvfp4", "nvfp4", 4096, 4096, 8, 128, 257, True), ("nvfp4", "fp8", 4096, 4096, 8, 128, 512, False),
    ("nvfp4", "fp8", 4096, 4104, 8, 128, 200, True), ("nvfp4", "fp8", 4096, 4096, 2, 256, 200, True),
    ("nvfp4", "fp8", 4096, 6144, 4, 16, 256, False), ("nvfp4", "fp8", 4096, 6144, 4, 32, 256, True),
    ("nvfp4", "fp8", 4096, 4096, 3, 16, 512, False), ("nvfp4", "fp8", 4096, 4096, 3, 16, 513, True),
    ("nvfp4", "bf16", 4096, 4096, 1, 16, 200, True), ("nvfp4", "bf16", 4096, 4096, 6, 256, 256, False),
    ("nvfp4", "bf16", 4096, 4096, 6, 256, 257, True), ("nvfp4", "bf16", 4096, 4096, 7, 256, 200, True),
    ("fp8", "fp8", 4096, 4096, 4, 16, 256, False), ("fp8", "fp8", 4096, 4096, 4, 16, 257, True), ("fp8", "fp8", 4096, 4096, 4, 32, 256, True),
    ("fp8", "nvfp4", 3696, 8192, 4, 128, 256, False), ("fp8", "nvfp4", 3696, 8200, 4, 128, 256, True),
    ("fp8", "nvfp4", 3696, 8192, 2, 128, 256, True), ("fp8", "nvfp4", 3696, 8192, 4, 128, 257, True),
    ("fp8", "fp8", 4096, 4096, 6, 256, 300, False), ("fp8", "fp8", 4096, 4096, 7, 256, 300, True), ("fp8", "bf16", 4096, 4096, 6, 256, 200, True)])
def test_which_stored_adapters_keep_the_small_tiles(base, fmt, K, N, L, R, M, large):
    """Either side of each line of the rule, and the same output to rounding whichever way: within 2e-2 of ||y||inf of the route that
    is asked for by name (both against the oracle: above, and test_token_tiles_gpu.py)."""
    d = configs.draw(K, (N,), R, L, M, seed=R + M, ids_low=-1, w_std=0.05, b_std=0.05)
    op = (build_fp8_op(configs.with_fp8_base(d), max_m=M, lora_fp8=fmt == "fp8", lora_fp4=fmt == "nvfp4") if base == "fp8"
          else build_nvfp4_op(configs.with_nvfp4_base(d), max_m=M, lora_fmt=fmt))
    assert [op.resolved_tile(M, c)["prefill"] for c in (None, {"prefill": 1}, {"prefill": 2})] == [1 if large else 2, 1, 2]
    meta, x = device_meta(make_index(d["ids"], L, M), M), d["x"].cuda()
    y, other = op(x, meta), op(x, meta, cfg={"prefill": 2 if large else 1})
    torch.cuda.synchronize()
    assert op.scratch.status()[0] == 0
    assert max_err_ratio(y, other.float().cpu()) <= TOL
