"""Memory ordering that no run can be made to violate on purpose, checked in the source: in a CTA pair, one CTA's threads write
operand tiles to their shared memory and a thread of the OTHER CTA issues the MMA that reads them, so the arrival that publishes
the tiles must release at cluster scope (a CTA-scope release does not synchronize with a thread of another CTA)."""
from __future__ import annotations

import re
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "onebase_b200" / "csrc"


def _ptx_of(helper: str) -> str:
    text = (CSRC / "ob_ptx.cuh").read_text()
    body = re.search(r"void " + helper + r"\(uint32_t cluster_addr\) \{(.*?)\n\}", text, re.S)
    assert body, helper
    return body.group(1)


def test_converted_operand_tiles_are_published_at_cluster_scope():
    text = (CSRC / "k2_prefill2.cu").read_text()
    helpers = re.findall(r"(\w+)\(cluster_peer_addr\(smem_u32\(&ctrl->conv\[", text)
    assert helpers
    for helper in helpers:
        assert "mbarrier.arrive.release.cluster." in _ptx_of(helper), helper
