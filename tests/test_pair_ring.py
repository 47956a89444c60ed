"""The weight ring of the ternary product on CTA pairs: csrc/gemm_tc_pair_walk.h, the order in which the kernel's unpack groups wait for weight loads and
hand them back, under many schedules on the CPU.  K of one to fourteen blocks and of 54 (a last load of 1, 2, 3 and 4 blocks), one tile and several, both depths
of the operand ring."""
import subprocess
from pathlib import Path

import pytest

HERE = Path(__file__).resolve().parent
CSRC = HERE.parent / "wrinklefree-inference-engine_b200" / "csrc"


@pytest.fixture(scope="module")
def ring(tmp_path_factory):
    exe = tmp_path_factory.mktemp("ring") / "pair_ring"
    subprocess.run(["/usr/bin/g++", "-O1", "-std=c++17", f"-I{CSRC}", str(HERE / "pair_ring.cpp"), "-o", str(exe)], check=True)

    def run(kb, tiles, stages, seeds, form):
        out = subprocess.run([str(exe), *map(str, (kb, tiles, stages, seeds, form))], check=True, capture_output=True, text=True, timeout=120).stdout.split()
        return int(out[1]), int(out[3])
    return run


@pytest.mark.parametrize("stages", [4, 8])
@pytest.mark.parametrize("kb", [*range(1, 15), 54])
def test_no_group_reads_a_load_that_has_not_landed(ring, kb, stages):
    for tiles in (1, 2, 5):
        assert ring(kb, tiles, stages, 300, 0) == (0, 0), tiles


def test_the_schedules_find_a_load_left_out(ring):
    """The same ring with groups that skip the loads without an item of theirs reads codes of the load before: the schedules above do reach that."""
    assert sum(ring(kb, 5, stages, 300, 1)[0] for kb in (5, 6, 54) for stages in (4, 8)) > 0
