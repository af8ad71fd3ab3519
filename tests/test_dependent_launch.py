"""Kernels of the drivers' dependent launches: each starts with the wait for the
kernel before it, and none reads an array by a load that promises the data does
not change while the kernel is resident (the kernel before it may still write)."""
import glob
import os
import re

from lsmlib_b200 import build

TEXT = {os.path.basename(f): re.sub(r"//[^\n]*", "", open(f).read())
        for f in glob.glob(os.path.join(build.CSRC, "*.cu*"))}


def closing(text, at):
    """The index of the bracket that closes the one at ``at``."""
    pair = {"(": ")", "{": "}"}[text[at]]
    depth = 0
    for i in range(at, len(text)):
        depth += {text[at]: 1, pair: -1}.get(text[i], 0)
        if depth == 0:
            return i
    raise AssertionError("unbalanced")


def device_functions():
    """Function name -> bodies: the kernels and device functions."""
    found = {}
    for text in TEXT.values():
        for m in re.finditer(r"\b(\w+)\(", text):
            end = closing(text, m.end() - 1)
            body = re.match(r"\s*(?:const\s*)?\{", text[end + 1:])
            head = re.split(r"[;{}]", text[:m.start()])[-1]
            if body and ("__global__" in head or "__device__" in head):
                start = end + body.end()
                found.setdefault(m.group(1), []).append(
                    text[start + 1:closing(text, start)].strip())
    return found


BODY = device_functions()


def launched():
    names = set()
    for text in TEXT.values():
        names |= set(re.findall(r"launch_after\(\(?(k_\w+)", text))
    return names


def reached(name, seen):
    """The bodies of a kernel and of every device function it may call."""
    if name in seen:
        return
    seen.add(name)
    for body in BODY.get(name, []):
        yield name, body
        local = set(re.findall(r"\bauto (\w+) = \[", body))   # lambdas
        for callee in set(re.findall(r"\b(\w+)\s*(?:<[^;(){}]*>)?\(", body)) - local:
            if callee in BODY:
                yield from reached(callee, seen)


def test_every_dependent_kernel_waits_first():
    names = launched()
    assert {"k_stage_pairs", "k_stage_pairs_up", "k_face_ghosts", "k_rk", "k_adjoint_stage",
            "k_deform_g"} <= names
    for name in names:
        assert BODY[name] and all(b.startswith("grid_wait();") for b in BODY[name]), name


def test_no_loads_of_constant_data():
    seen = set()
    for name in launched():
        for inner, body in reached(name, seen):
            for word in ("__ldg", "__restrict__", "ld.global.nc"):
                assert word not in body, (name, inner, word)
    assert {"stage_tile_pairs", "stage_tile_pairs_up", "face_ghost_value", "stage_out",
            "weno5_face2", "weno5_side_fast"} <= seen
