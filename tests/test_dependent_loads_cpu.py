"""Loads of the device code that run in kernels started ahead of their predecessors'
end (programmatic dependent launch), checked in the source: such a kernel is alive while
another one writes what it reads after its wait, so its loads must be coherent ones
(never ld.global.nc) and must not be movable above the wait (volatile statements)."""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "haissinskijulia_b200" / "csrc"
SOURCES = sorted(CSRC.glob("*.cu")) + sorted(CSRC.glob("*.cuh")) + sorted(CSRC.glob("*.h"))


def _code(path):
    text = re.sub(r"/\*.*?\*/", "", path.read_text(), flags=re.S)
    return re.sub(r"//[^\n]*", "", text)


def test_inline_loads_are_coherent_and_ordered():
    seen = 0
    for path in SOURCES:
        for m in re.finditer(r"asm\s*(volatile)?\s*\(\s*\"(ld\.global[^ ]*)", _code(path)):
            seen += 1
            assert m.group(1), (path.name, m.group(2))
            assert ".nc" not in m.group(2), (path.name, m.group(2))
    assert seen >= 4


def test_the_pass_reads_through_no_non_coherent_intrinsic():
    code = _code(CSRC / "hj_track.cu")
    body = code[code.index("void pass_body("):code.index("k_batch_pass(")]
    assert "grid_dependency_wait" in body and "__ldg" not in body


def test_the_scan_reads_ahead_of_its_wait_past_l1():
    code = _code(CSRC / "hj_scan.cu")
    early = code[code.index("void scan_body("):]
    early = early[:early.index("grid_dependency_wait()")]
    assert "load_scalars(&ts->cur)" in early
    assert "ts->" not in early.replace("&ts->cur", "")
    assert "__ldcg" in code[code.index("load_scalars("):code.index("void scan_body(")]
