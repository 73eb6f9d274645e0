"""Kernels of a frame start while their predecessor drains and wait for its writes at entry.  A
read-only load (__ldg) is for memory that nothing writes while the kernel runs and is not ordered
by that wait, so nothing that a frame's kernels write is read with one."""
import re
from pathlib import Path

SRC = Path(__file__).resolve().parents[1] / "master-of-puppets_b200" / "csrc" / "kernels.cu"
READ_ONLY = {"sky", "irr", "pf", "brdf"}  # a frame's inputs among FrameArgs' pointers


def test_no_read_only_load_of_what_a_frame_writes():
    src = SRC.read_text()
    members = re.findall(r"__ldg\(\s*(?:\([^()]*\)\s*)?&?\(?a\.(\w+)", src)
    assert members, "the pattern finds the loads of the inputs"
    assert set(members) <= READ_ONLY, sorted(set(members) - READ_ONLY)
