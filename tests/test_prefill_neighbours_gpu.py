"""The fused neighbours on the large-tile prefill path: silu(gate) * up formed by the quantizing kernels (row in registers up
to 4096 and 12288 elements, in two passes beyond, and the NVFP4 form) and the residual stream added in the CTA-pair GEMM's
stores (in place and not, a ragged last token tile, several tiles per pair)."""
from __future__ import annotations

import pytest
import torch

from helpers import build_fp8_op, build_nvfp4_op, device_meta, make_index
from oracle import configs, neighbours as onb, nvfp4 as on4

pytestmark = pytest.mark.gpu


def _op(base, K, widths, R, L, M, x=None):
    d = configs.draw(K, widths, R, L, M, seed=K + M, ids_low=-1, w_std=0.05, b_std=0.05)
    d["ids"] = configs.zipf_request_ids(M, L, seed=2, mean_len=40)
    d["ids"][5:17] = -1
    if base == "fp8":
        return d, build_fp8_op(configs.with_fp8_base(d), max_m=M)
    d = configs.with_nvfp4_base(d)
    if x is not None:
        d["x_global"] = on4.global_scale_for(x.float())
    return d, build_nvfp4_op(d, max_m=M)


@pytest.mark.parametrize("base,K", [("fp8", 4096), ("fp8", 4112), ("fp8", 12288), ("fp8", 14784), ("nvfp4", 4096)])
def test_silu_mul_of_a_prefill_batch(base, K):
    M, widths = 515, (512,)
    g = torch.Generator().manual_seed(K)
    gu = (torch.randn(M, 2 * K, generator=g) * 1.5).to(torch.bfloat16)
    act = onb.silu_mul(gu)
    d, op = _op(base, K, widths, 64, 4, M, act)
    meta = device_meta(make_index(d["ids"], 4, M), M)
    y = op(gu.cuda(), meta, silu_mul=True).float()
    y_plain = op(act.cuda(), meta).float()
    torch.cuda.synchronize()
    assert op.scratch.status()[0] == 0
    # the two routes differ only where the device's and the host's expf flipped a bf16 rounding of the activation
    assert float((y - y_plain).abs().max() / y_plain.abs().max()) <= 4e-3
    assert float((y != y_plain).float().mean()) < 0.05


@pytest.mark.parametrize("base,widths", [("fp8", (512, 1024)), ("nvfp4", (256, 512)), ("fp8", (20480,))])
@pytest.mark.parametrize("in_place", [False, True])
def test_residual_of_a_prefill_batch(base, widths, in_place):
    M, K, L = 1037, 1024, 6
    N = sum(widths)
    d, op = _op(base, K, widths, 64, L, M)
    meta = device_meta(make_index(d["ids"], L, M), M)
    x = d["x"].cuda()
    res = torch.randn(M, N, generator=torch.Generator().manual_seed(3)).to(torch.bfloat16)
    y_plain = op(x, meta).clone()
    want = onb.add_residual(y_plain.cpu(), res)                # bf16(y) + residual in fp32, one rounding: exact
    r_dev = res.cuda()
    y = op(x, meta, out=r_dev if in_place else None, residual=r_dev)
    torch.cuda.synchronize()
    assert op.scratch.status()[0] == 0
    assert torch.equal(y.cpu(), want)
    # a residual the 16-byte loads cannot take goes to the small tiles
    r_odd = torch.empty(M, N + 4, dtype=torch.bfloat16, device="cuda")[:, 4:]
    r_odd.copy_(res)
    y_odd = op(x, meta, residual=r_odd)
    assert float((y_odd.float().cpu() - want.float()).abs().max() / want.float().abs().max()) <= 2e-2


@pytest.mark.parametrize("base,widths", [("fp8", (512, 264)), ("nvfp4", (256, 520)), ("fp8", (20480,))])
@pytest.mark.parametrize("fmt", ["fp8", "nvfp4"])
def test_residual_of_a_prefill_batch_with_stored_adapters(base, widths, fmt):
    M, K, L = 1037, 512, 6
    N = sum(widths)
    d, _ = _op(base, K, widths, 64, L, M)
    op = (build_fp8_op(d, max_m=M, lora_fp8=fmt == "fp8", lora_fp4=fmt == "nvfp4") if base == "fp8"
          else build_nvfp4_op(d, max_m=M, lora_fmt=fmt))
    meta = device_meta(make_index(d["ids"], L, M), M)
    x = d["x"].cuda()
    res = torch.randn(M, N, generator=torch.Generator().manual_seed(3)).to(torch.bfloat16)
    want = onb.add_residual(op(x, meta).cpu(), res)            # (the plain output against the oracle: test_prefill_stored_gpu.py)
    y = op(x, meta, residual=res.cuda())
    torch.cuda.synchronize()
    assert op.scratch.status()[0] == 0
    assert torch.equal(y.cpu(), want)
