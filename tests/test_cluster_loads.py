"""A bulk load that one CTA issues for a whole cluster must never meet another GPU's memory, and the kernels here also run in tensor-parallel processes:
no source issues one (commits that signal several CTAs' barriers are another matter)."""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parents[1] / "wrinklefree-inference-engine_b200" / "csrc"


def test_no_bulk_load_is_shared_by_a_cluster():
    found = []
    for p in sorted(CSRC.rglob("*.cu*")):
        for i, line in enumerate(p.read_text().splitlines(), 1):
            if re.search(r"cp\.async\.bulk\S*multicast", line) or re.search(r"SM\d+_TMA_LOAD_MULTICAST", line):
                found.append(f"{p.name}:{i}")
    assert not found, found
