"""A bulk load that one CTA issues for a whole cluster must never meet another GPU's memory, and the kernels here also run in tensor-parallel processes:
every bulk copy in the sources is one of the forms that serve the issuing CTA (or pair) alone."""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parents[1] / "wrinklefree-inference-engine_b200" / "csrc"
QUALIFIERS = {"cp", "async", "bulk", "tensor", "1d", "2d", "3d", "4d", "5d", "prefetch", "L2", "global", "shared::cluster", "shared::cta", "mbarrier::complete_tx::bytes",
              "cta_group::1", "cta_group::2", "commit_group", "wait_group", "read", "bulk_group"}


def test_bulk_copies_serve_the_cta_that_issues_them():
    found, seen = [], 0
    for p in sorted(CSRC.rglob("*.cu*")):
        for i, line in enumerate(p.read_text().splitlines(), 1):
            for name in re.findall(r'"[^"]*?(cp\.async\.bulk[\w.:]*)', line):
                seen += 1
                extra = set(name.split(".")) - QUALIFIERS
                if extra:
                    found.append((f"{p.name}:{i}", extra))
    assert seen and not found, found
