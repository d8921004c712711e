"""The segment index over the edges of its work split: fewer tokens than a warp's group of 32, tokens beyond the ones a warp
keeps in registers (8192), the sizes at which a batch takes one more warp, ragged last chunks, and slot counts around the points where fewer warps share the histogram
(309 | 310 slots, and the largest 1023); all five tensors bit-equal to the oracle."""
from __future__ import annotations

import pytest
import torch

from oracle import segments as oseg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L", [1, 32, 309, 310, 1023])
@pytest.mark.parametrize("M", [1, 31, 33, 64, 65, 129, 256, 257, 513, 1023, 1025, 4097, 8192, 8193, 20011])
def test_segment_index_equals_oracle(M, L):
    from onebase_b200.metadata import KernelMeta
    g = torch.Generator().manual_seed(M * 7 + L)
    ids = torch.randint(-1, L, (M,), generator=g, dtype=torch.int32)
    if M > 100:
        ids[40:90] = 0                                        # a run of one tenant across a group's edge
    ids[0] = 0                                                # at least one adapter
    ref = oseg.SegmentIndex(L, M)
    ref.prepare(ids)
    given = ids.clone()
    km = KernelMeta.make(L, M, "cuda")
    km.prepare_tensors(given.cuda())
    tok, srt, seg_n, seg_start, seg_ids = (t.cpu() for t in km.meta_args(M))
    assert torch.equal(tok, ref.tok) and torch.equal(srt, ref.srt)
    assert torch.equal(seg_n, ref.seg_n) and torch.equal(seg_start, ref.seg_start) and torch.equal(seg_ids, ref.seg_ids)
    km.prepare_tensors(torch.full((M,), -1, dtype=torch.int32, device="cuda"))   # no adapter: the sort stays, the segments empty
    assert torch.equal(km.token_indices_sorted_by_lora_ids.cpu(), ref.srt) and int(km.num_tokens_per_lora.sum()) == 0
