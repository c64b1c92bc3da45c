"""Warp votes and shuffles name lanes that provably arrive together: the mask that
__activemask() returns is whatever lanes the scheduler runs at that moment, which says
nothing about the next instruction."""
from pathlib import Path

CSRC = Path(__file__).resolve().parents[1] / "pecs_gb300" / "csrc"


def test_no_mask_of_the_moment():
    files = [f for f in CSRC.iterdir() if f.suffix in (".cu", ".cuh")]
    assert len(files) > 5
    assert [f.name for f in files if "__activemask" in f.read_text()] == []
