"""The adjoint's reverse sweep reads every state's ghost cells as stored, so its
forward stages store them themselves and leave nothing to the kernel that a stage
happens to run in (the one-cell kernel makes boundary values without storing them)."""
import os
import re

from lsmlib_b200 import build


def body(text, head):
    start = text.index("{", text.index(head))
    depth = 0
    for at in range(start, len(text)):
        depth += {"{": 1, "}": -1}.get(text[at], 0)
        if depth == 0:
            return text[start:at]


def test_forward_stage_stores_ghost_cells():
    text = open(os.path.join(build.CSRC, "adjoint.cu")).read()
    stage = body(text, "cudaError_t fwd_stage(")
    assert re.search(r"launch_ghosts\(8, a, st\).*bc_mask = 0u.*launch_stage_fast\(", stage, re.S)
    # the only launch of a forward stage
    assert text.count("launch_stage_fast(") == 1
    assert "ghosts_writable" not in text
