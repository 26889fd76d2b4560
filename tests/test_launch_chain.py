"""CPU check of the step's chain of launches (csrc/launch.cuh, launch_after): a kernel launched so
may start before the one ahead of it has finished, so it begins by waiting (begin_after), and no
load of what the chain writes may come before the wait.  Every such kernel hands its __restrict__
pointers to begin_after, and the tool's segments and the sort's slots, which reach a kernel inside
a struct, are not read by non-coherent loads."""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parents[1] / "sph_fem_2d_cutting_gpu_gb300" / "csrc"
SOURCES = {p.name: p.read_text() for p in sorted(CSRC.glob("*.cu*"))}


def kernels():
    """name -> (parameters, first statement of the body)"""
    out = {}
    for text in SOURCES.values():
        for m in re.finditer(r"__global__[^{;]*?\b(k_\w+)\s*\(([^{;]*?)\)\s*\{\s*([^;]*;)", text):
            out[m.group(1)] = (" ".join(m.group(2).split()).split(","), m.group(3))
    return out


def launched():
    names = set()
    for text in SOURCES.values():
        for m in re.finditer(r"launch_after\(s, *(.*?);", text, re.S):
            names |= set(re.findall(r"\bk_\w+", m.group(1)))
    return names


def test_chained_kernels_wait_first():
    known = kernels()
    assert len(launched()) > 15 and launched() <= set(known)
    for name in launched():
        parameters, first = known[name]
        begin = re.fullmatch(r"begin_after\((.*)\);", first)
        assert begin, f"{name} starts with: {first}"
        restricted = {re.search(r"(\w+)$", p.strip()).group(1) for p in parameters if "__restrict__" in p}
        handed = {p.strip() for p in begin.group(1).split(",") if p.strip()}
        assert handed == restricted, (name, restricted - handed)


def test_no_non_coherent_loads_of_struct_members():
    for name, text in SOURCES.items():
        for line in text.splitlines():
            assert not re.search(r"__ldg\((seg|X|A|B|F|K)\.|__ldg\(slots", line), (name, line.strip())
