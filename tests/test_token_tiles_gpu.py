"""An explicit token tile narrower than the batch: many 16- or 32-token tiles, whose GEMM takes h from the warp-level shrink's
fp32 partials, over both bases and all three adapter storages -- outputs within 2e-2 * ||y||inf of the oracle on the adapters as
stored, from a workspace whose partials hold something else before the call."""
from __future__ import annotations

import pytest
import torch

from helpers import build_fp8_op, build_nvfp4_op, device_meta, make_index, max_err_ratio, stored_adapters
from oracle import configs, fp8 as ofp8, nvfp4 as on4

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("base", ["fp8", "nvfp4"])
@pytest.mark.parametrize("fmt", ["bf16", "fp8", "nvfp4"])
@pytest.mark.parametrize("M,cfg", [(200, {"tn": 16}), (200, {"tn": 32}), (600, {"tn": 16}), (600, {"tn": 32}),
                                   (200, {"tn": 32, "prefill": 1}), (40, {"tn": 32, "prefill": 1})])
def test_many_small_token_tiles(base, fmt, M, cfg):
    K, widths, R, L = 512, (264, 120), 64, 6
    d = configs.draw(K, widths, R, L, M, seed=M, ids_low=-1, w_std=0.05, b_std=0.05)
    if base == "fp8":
        d = configs.with_fp8_base(d)
        op = build_fp8_op(d, max_m=M, lora_fp8=fmt == "fp8", lora_fp4=fmt == "nvfp4")
    else:
        d = configs.with_nvfp4_base(d)
        op = build_nvfp4_op(d, max_m=M, lora_fmt=fmt)
    assert op.resolved_tile(M, cfg)["prefill"] == 2
    op.scratch.region("hp", op.scratch.sizes["hp"]).view(torch.float32).fill_(3.0)
    y = op(d["x"].cuda(), device_meta(make_index(d["ids"], L, M), M), cfg=cfg)
    torch.cuda.synchronize()
    assert op.scratch.status()[0] == 0, op.scratch.status()[:8]
    A, B = stored_adapters(op, fmt)
    if base == "fp8":
        ref = ofp8.fused_projection(d["x"], d["ids"], d["w_q"], d["s_w"], A, B, widths)
    else:
        ref = on4.fused_projection(d["x"], d["ids"], d["w_q4"], d["w_sf"], d["w_global"], d["x_global"], A, B, widths)
    assert max_err_ratio(y, ref) <= 2e-2
