"""Warp votes, shuffles and reductions of the kernels name their lanes from
values that all of them hold (the group's mask, chunk_mask): the set that
__activemask() reports is whatever happens to be converged, which CUDA does not
promise to keep until the next instruction."""
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "scream_gb300" / "csrc"


def test_no_collective_under_the_active_mask():
    for src in sorted(CSRC.glob("*.cu*")):
        assert "__activemask" not in src.read_text(), src.name
