"""Barriers of a part of a block in the CUDA sources: the instruction is defined for warps whose lanes arrive together, so
nothing but the helper that brings them together first (part_barrier) may issue it."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "amca3d_gb300", "csrc")


def test_every_barrier_of_part_of_a_block_follows_a_warp_barrier():
    uses = 0
    for name in sorted(os.listdir(CSRC)):
        if not name.endswith((".cu", ".cuh", ".h")):
            continue
        src = open(os.path.join(CSRC, name)).read()
        for m in re.finditer(r'asm volatile\("(bar|barrier)(\.cta)?\.(sync|red|arrive)', src):
            before = [line.strip() for line in src[:m.start()].splitlines() if line.strip()]
            assert before[-1] == "__syncwarp();", (name, src.count("\n", 0, m.start()) + 1)
            uses += 1
    assert uses >= 1
