"""Kernels whose launch overlaps the one before them (launch_pdl, griddepcontrol): what that kernel writes may change while they are resident, so it is waited for and read
with ordinary loads.  Read from the sources: the non-coherent loads (`__ldg`, `const ... __restrict__` parameters) are left to weights, which no kernel of the chain
writes."""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parents[1] / "wrinklefree-inference-engine_b200" / "csrc"
SOURCES = sorted(CSRC.rglob("*.cu"))
# packed or dense weights and a bias table: (file, what is loaded)
WEIGHTS = {("gemm_tc.cu", "l_src"), ("gemv_packed.cu", "wr"), ("seq_gemm.cu", "wa"), ("seq_gemm.cu", "wb"), ("seq_attn_mma.cu", "D.rel")}


def kernels(text):
    """name -> (parameters, body up to the next kernel)"""
    starts = [m.start() for m in re.finditer(r"__global__", text)] + [len(text)]
    out = {}
    for a, b in zip(starts, starts[1:]):
        m = re.match(r"__global__\s+void\s+(?:__launch_bounds__\((?:[^()]|\([^()]*\))*\)\s*)?(?:__cluster_dims__\([^()]*\)\s*)?(\w+)\s*\(", text[a:b])
        assert m, text[a:a + 120]
        end = text.index(")", a + m.end())
        while text[a:end + 1].count("(") != text[a:end + 1].count(")"):
            end = text.index(")", end + 1)
        out[m.group(1)] = (text[a + m.end():end], text[end:b])
    return out


def overlapped():
    """(file, kernel, parameters, body) of every kernel that is launched ahead of its predecessor's end"""
    for p in SOURCES:
        text = p.read_text()
        for name, (params, body) in kernels(text).items():
            if re.search(r"pdl_enter\(\)|pdl_wait_prior\(\)", body):
                yield p.name, name, params, body


def test_every_launch_that_overlaps_waits():
    waiting = {name for _, name, _, _ in overlapped()}
    launched = set()
    for p in SOURCES:
        launched |= set(re.findall(r"launch_(?:pdl|rows)\(\s*(\w+)", p.read_text())) - {"kern"}
    assert len(launched) > 40 and launched <= waiting, launched - waiting


def test_results_of_the_kernel_before_are_read_coherently():
    found = []
    for file, name, params, body in overlapped():
        if file in ("glue.cu",):                      # embedding, head and argmax of the decode engine: launched behind the end of the kernel before
            continue
        found += [(file, name, x) for x in re.findall(r"const [^,]*__restrict__ \w+", params)]
    for p in SOURCES:
        for x in re.findall(r"__ldg\(([^;]*)", p.read_text()):
            what = re.search(r"(?:reinterpret_cast<[^>]*>\()?\(?([\w.]+)", x).group(1)
            if (p.name, what) not in WEIGHTS:
                found.append((p.name, "__ldg", x[:40]))
    assert not found, found
