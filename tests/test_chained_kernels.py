"""Kernels whose CTAs may be placed while the kernel in front of them drains: no load of theirs may be moved in front of their wait.  A compiler may do that
with what it knows to be constant (const __restrict__ parameters, __ldg, ld.global.nc), so the sources hold none of it that is not made behind the wait."""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "koboldcpp_b200" / "csrc"
# device code that only chained kernels call
HELPERS = ("mmvq_core.cuh", "mmvq3.cuh", "mmvq_mma.cuh", "fattn_mma.cuh", "fattn_tc.cuh", "sink_tile.cuh", "rope_kv.cuh")


def kernels():
    for path in sorted(CSRC.glob("*.cu")) + sorted(CSRC.glob("*.cuh")):
        parts = re.split(r"(?=__global__)", re.sub(r"//.*", "", path.read_text()))[1:]
        for part in parts:
            head, _, body = part.partition("{")
            if "pdl_enter(" in body or "pdl_wait(" in body:
                yield path.name, head, body


def test_constant_pointers_are_made_behind_the_wait():
    found = 0
    for name, head, body in kernels():
        found += 1
        pointers = re.findall(r"const \w[\w ]*\*\s*__restrict__\s*(\w+)", head)
        tied = re.search(r"pdl_enter\(([^)]*)\)", body)
        missing = set(pointers) - set(re.findall(r"\w+", tied.group(1)) if tied else [])
        assert not missing, (name, re.search(r"(\w+)\(", head[head.index("void"):]).group(1), missing)
    assert found >= 20


def test_no_load_of_constant_memory():
    for name, head, body in kernels():
        assert "__ldg(" not in body and "ld.global.nc" not in body, (name, head[:120])
    for name in HELPERS:
        text = re.sub(r"//.*", "", (CSRC / name).read_text())
        assert "__ldg(" not in text and "ld.global.nc" not in text, name


def test_loads_from_a_peers_shared_memory_stay_between_the_cluster_barriers():
    """A compiler may move an asm without volatile across a barrier, whose clobber holds ordinary loads and volatile ones."""
    found = 0
    for path in sorted(CSRC.glob("*.cu*")):
        for keyword in re.findall(r"(asm(?: volatile)?)\s*\(\s*\"ld\.shared::cluster", path.read_text()):
            found += 1
            assert keyword == "asm volatile", path.name
    assert found
