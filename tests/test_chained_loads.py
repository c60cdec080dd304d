"""Kernels that may be launched chained (they call chainBegin and exist while the
kernel before them writes) read what other kernels of a step write with ordinary
loads: every __ldg in them, and in the device functions they call, is of a table
that no kernel of a step writes.  Read off the sources."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "behavert_b200" / "csrc"
TABLES = {"agentBase", "obstacles", "obsMask", "tiles"}
FILES = ["brt_internal.cuh", "brt_agent.cuh", "brt_order.cu", "brt_fused.cu", "brt_school.cu", "brt_kernels.cu", "brt_adjoint.cu"]
# device functions that no chained kernel calls: the per-agent scans (flockKernel
# asserts it), the crowd stage's separation and the tile kernel's scan
UNCHAINED = {"scanNeighborsFlat", "scanNeighborsPipelined", "separationDir", "scanTileStaged"}


def _parts(text):
    """The file cut after every top-level closing brace, without comments."""
    return re.split(r"\n}\n", re.sub(r"//[^\n]*", "", text))


def _name(part):
    m = re.search(r"(?:__forceinline__|__global__|static|inline)[^;{=]*?\b(\w+)\(", re.sub(r"__launch_bounds__\([^)]*\)", "", part))
    return m.group(1) if m else ""


PARTS = [(f, _name(p), p) for f in FILES for p in _parts((CSRC / f).read_text())]
CHAINED = [x for x in PARTS if "__global__" in x[2] and "chainBegin()" in x[2]]
LOADERS = {n for _, n, p in PARTS if "template <bool CHAIN" in p and "__global__" not in p}


@pytest.mark.parametrize("name", FILES)
def test_only_tables_by_non_coherent_loads(name):
    for f, fn, part in PARTS:
        if f != name or ("__global__" in part and "chainBegin()" not in part) or fn in UNCHAINED or "T ldStep(" in part:
            continue
        assert set(re.findall(r"__ldg\(\s*&?\s*(?:\w+\.)?(\w+)", part)) <= TABLES, fn


def test_chained_kernels_choose_ordinary_loads():
    assert len(CHAINED) >= 9 and len(LOADERS) >= 10
    for _, fn, part in CHAINED + [x for x in PARTS if x[1] in LOADERS]:
        for callee in LOADERS:
            for arg in re.findall(r"\b%s<(\w+)" % callee, part):
                assert arg in ("CHAIN", "true"), (fn, callee, arg)
        for callee in UNCHAINED - {"scanNeighborsFlat", "scanNeighborsPipelined"}:
            assert callee + "(" not in part, (fn, callee)


def test_launches():
    """The first kernel of launchChainedOr is the chained instantiation, and what
    launchChained takes reads by ordinary loads whatever the size."""
    text = "".join(p for _, _, p in PARTS)
    pairs = re.findall(r"launchChainedOr\(A\.n,\s*(\w+)<([^>()]*(?:\([^)]*\))?[^>()]*)>,\s*(\w+)<([^>()]*(?:\([^)]*\))?[^>()]*)>", text)
    assert {p[0] for p in pairs} == {"countKernel", "placeKernel", "reorderKernel", "fusedKernel", "schoolKernel", "flockKernel"}
    for a, chained, b, plain in pairs:
        assert a == b and chained.endswith("true"), (a, chained)
        assert plain != chained
    singles = set(re.findall(r"launchChained\(A\.n,\s*(\w+<[^>]*>)", text))
    assert singles == {"cellScanKernel<256, 1>", "cellScanKernel<256, 2>", "cellScanKernel<256, 4>", "cellScanKernel<1024, 8>",
                       "adjointStepKernel<4>", "adjointGatherKernel<4>", "adjointGatherKernel<8>"}
    step = next(p for _, fn, p in CHAINED if fn == "adjointStepKernel")
    assert "constexpr bool CHAIN = LANES == 4;" in step
    gather = next(p for _, fn, p in CHAINED if fn == "adjointGatherKernel")
    assert "ldStep<true>" in gather and "ldStep<CHAIN>" not in gather
    flock = next(p for _, fn, p in CHAINED if fn == "flockKernel")
    assert "static_assert(!CHAIN || SCAN >= 4" in flock
