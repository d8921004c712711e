"""The CTA-pair prefill GEMM over the layers it takes since slices need not be whole tiles: widths that end anywhere in a tile
(in steps of 8 features), ranks below and above one 64-rank expand step, both bases, batches from the first size it serves
(129 tokens) on, tenants that cross the edge of a 128-token block (one expand step for both blocks) and tokens without an
adapter -- outputs within 2e-2 * ||y||inf of the oracle's fp32 result, the large tiles asserted to be what ran."""
from __future__ import annotations

import pytest
import torch

from helpers import build_fp8_op, build_nvfp4_op, device_meta, make_index, max_err_ratio, oracle_y, oracle_y_nvfp4, stored_adapters
from oracle import configs, fp8 as ofp8

pytestmark = pytest.mark.gpu
TOL = 2e-2

CASES = [("fp8", 512, (264, 120, 1000), 16, 5, 129), ("fp8", 528, (3696,), 32, 40, 300), ("fp8", 256, (512, 8), 64, 3, 257),
         ("fp8", 1024, (776,), 128, 7, 517), ("fp8", 512, (256, 256), 256, 2, 1000), ("fp8", 512, (4096, 24576), 64, 8, 777),
         ("nvfp4", 512, (264, 120, 1000), 16, 5, 129), ("nvfp4", 1024, (3696,), 32, 40, 300), ("nvfp4", 512, (776, 136), 64, 7, 517),
         ("nvfp4", 256, (384,), 128, 3, 1000)]


@pytest.mark.parametrize("base,K,widths,R,L,M", CASES)
def test_pair_gemm_ragged_slices_and_ranks(base, K, widths, R, L, M):
    d = configs.draw(K, widths, R, L, M, seed=K + M + R, ids_low=-1, w_std=0.05, b_std=0.05)
    d["ids"] = configs.zipf_request_ids(M, L, seed=M, mean_len=50)
    d["ids"][60:75] = -1
    if base == "fp8":
        d = configs.with_fp8_base(d)
        op, ref = build_fp8_op(d, max_m=M), oracle_y(d, d["x"], d["ids"])
    else:
        d = configs.with_nvfp4_base(d)
        op, ref = build_nvfp4_op(d, max_m=M), oracle_y_nvfp4(d, d["x"], d["ids"])
    assert op.resolved_tile(M)["prefill"] == 1
    meta = device_meta(make_index(d["ids"], L, M), M)
    y = op(d["x"].cuda(), meta)
    y2 = op(d["x"].cuda(), meta, out=torch.full_like(y, 7.0))
    torch.cuda.synchronize()
    assert op.scratch.status()[0] == 0, op.scratch.status()[:8]
    assert max_err_ratio(y, ref) <= TOL and torch.equal(y, y2)


def test_an_unaligned_output_keeps_the_small_tiles():
    M, K, widths, L = 200, 512, (264, 120), 4
    d = configs.with_fp8_base(configs.draw(K, widths, 64, L, M, seed=1, ids_low=-1, w_std=0.05, b_std=0.05))
    op = build_fp8_op(d, max_m=M)
    out = torch.full((M, 384 + 3), 7.0, dtype=torch.bfloat16, device="cuda")
    op(d["x"].cuda(), device_meta(make_index(d["ids"], L, M), M), out=out[:, 1:385])
    torch.cuda.synchronize()
    assert op.scratch.status()[0] == 0
    assert max_err_ratio(out[:, 1:385], oracle_y(d, d["x"], d["ids"])) <= TOL
    assert bool((out[:, 0] == 7).all()) and bool((out[:, 385:] == 7).all())


@pytest.mark.parametrize("cfg", [{"prefill": 2}, {"prefill": 1, "tn": 64}])
def test_nvfp4_small_tiles_over_several_token_tiles(cfg):
    """The 64-token tiles, which the rule no longer takes at this size, with either shrink."""
    M, K, widths, L = 300, 1024, (264, 1000), 8
    d = configs.with_nvfp4_base(configs.draw(K, widths, 64, L, M, seed=8, ids_low=-1, w_std=0.05, b_std=0.05))
    op = build_nvfp4_op(d, max_m=M)
    y = op(d["x"].cuda(), device_meta(make_index(d["ids"], L, M), M), cfg=cfg)
    torch.cuda.synchronize()
    assert op.scratch.status()[0] == 0
    assert max_err_ratio(y, oracle_y_nvfp4(d, d["x"], d["ids"])) <= TOL


@pytest.mark.parametrize("widths,cfg", [((260,), None), ((264,), {"tn": 128})])
def test_the_tensor_core_shrink_starts_later_without_the_large_tiles(widths, cfg):
    """A layer (a slice that is no multiple of eight features) or a call (an explicit token tile) that the large tiles do not serve
    keeps the warp-level shrink up to the sizes where the tensor-core one is no slower in front of small tiles."""
    L, K, R = 4, 512, 16
    d = configs.with_fp8_base(configs.draw(K, widths, R, L, 1100, seed=2, ids_low=-1, w_std=0.05, b_std=0.05))
    for kw, first in (({}, 512), ({"lora_fp8": True}, 1024), ({"lora_fp4": True}, 1024)):
        op = build_fp8_op(d, max_m=1100, **kw)
        assert [op.resolved_tile(M, cfg)["prefill"] for M in (33, 129, first - 1, first)] == [2, 2, 2, 0]
        assert op.resolved_tile(129, {**(cfg or {}), "prefill": 1})["prefill"] == 0


@pytest.mark.parametrize("M", [200, 600])
@pytest.mark.parametrize("base,fmt", [("fp8", "bf16"), ("fp8", "nvfp4"), ("nvfp4", "bf16"), ("nvfp4", "fp8")])
def test_a_base_scaled_by_zero_leaves_the_adapters_term(base, fmt, M):
    """The large tiles add B h / s to the accumulator and scale by s: with s = 0 (a base of zeros, quantized by its largest value)
    y is the adapters' term alone, as on the smaller tiles."""
    K, widths, L = 512, (264, 120), 4
    d = configs.draw(K, widths, 32, L, M, seed=M, ids_low=-1, w_std=0.05, b_std=0.05)
    if base == "fp8":
        d = configs.with_fp8_base(d)
        d["s_w"] = torch.zeros(1)
        op = build_fp8_op(d, max_m=M, lora_fp8=fmt == "fp8", lora_fp4=fmt == "nvfp4")
    else:
        d = configs.with_nvfp4_base(d)
        op = build_nvfp4_op(d, max_m=M, lora_fmt=fmt)
        op.alpha.zero_()
    big = {"prefill": 1}
    assert op.resolved_tile(M, big)["prefill"] == 1
    y = op(d["x"].cuda(), device_meta(make_index(d["ids"], L, M), M), cfg=big)
    torch.cuda.synchronize()
    assert op.scratch.status()[0] == 0
    A, B = stored_adapters(op, fmt)
    assert max_err_ratio(y, ofp8.lora_term(d["x"], d["ids"], A, B, widths)) <= TOL
