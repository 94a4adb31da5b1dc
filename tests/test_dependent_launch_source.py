"""Kernels that may start before the one ahead of them has ended (pdl_wait) must not read
what it writes by the read-only path: that data is constant from a kernel's start on."""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parents[1] / "stimuli-responsive-nanodroplets_gb300" / "csrc"


def test_no_read_only_loads_beside_pdl_wait():
    seen = 0
    for src in sorted(CSRC.glob("*.cu")):
        text = re.sub(r"/\*.*?\*/|//[^\n]*", "", src.read_text(), flags=re.S)
        if "pdl_wait" not in text:
            continue
        seen += 1
        for word in ("__ldg", "ld.global.nc", "__restrict__"):
            assert word not in text, (src.name, word)
    assert seen >= 2
