"""Kernels of the drivers' dependent launches: each starts with the wait for the
kernel before it, and none reads an array by a load that promises the data does
not change while the kernel is resident (the kernel before it may still write)."""
import glob
import os
import re

from lsmlib_b200 import build

TEXT = {os.path.basename(f): re.sub(r"//[^\n]*", "", open(f).read())
        for f in glob.glob(os.path.join(build.CSRC, "*.cu*"))}


def kernel_body(name):
    for text in TEXT.values():
        m = re.search(r"__global__[^{;]*?\b%s\(" % name, text)
        if m:
            start = text.index("{", m.end())
            depth = 0
            for at in range(start, len(text)):
                depth += {"{": 1, "}": -1}.get(text[at], 0)
                if depth == 0:
                    return text[start + 1:at].strip()
    raise AssertionError("no kernel " + name)


def launched():
    names = set()
    for text in TEXT.values():
        names |= set(re.findall(r"launch_after\(\(?(k_\w+)", text))
    return names


def test_every_dependent_kernel_waits_first():
    names = launched()
    assert {"k_stage_pairs", "k_stage_pairs_up", "k_stage", "k_face_ghosts", "k_rk",
            "k_adjoint_stage", "k_deform_g"} <= names
    for name in names:
        assert kernel_body(name).startswith("grid_wait();"), name


def test_no_loads_of_constant_data():
    for name, text in TEXT.items():
        if "grid_wait();" not in text:
            continue
        for word in ("__ldg", "__restrict__", "ld.global.nc"):
            assert word not in text, (name, word)
    # (this file's other kernels may use the toolbox's read-only loads)
    assert not re.search(r"\bld\(", kernel_body("k_rk"))
