"""Kernels that begin with grid_wait() are resident while the launch before them
still writes the fields.  Their loads must therefore be ones that the compiler
keeps behind the wait and that are coherent: no __restrict__ field parameter, no
ld.global.nc, no __ldg of a field, volatile asm.  Shown on the sources: a load that
came too early would read links of the step before and raise no error."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "askja_b200", "csrc")


def source(path):
    text = re.sub(r"/\*.*?\*/", "", open(path).read(), flags=re.S)
    return re.sub(r"//[^\n]*", "", text)


def closing(text, i, pair):
    """Index of the bracket that closes the one at i."""
    depth = 0
    for j in range(i, len(text)):
        depth += (text[j] == pair[0]) - (text[j] == pair[1])
        if depth == 0:
            return j
    raise AssertionError("unbalanced")


def kernels():
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu*"))):
        text = source(path)
        for m in re.finditer(r"__global__", text):
            i = m.end()
            b = re.compile(r"\s*void\s*__launch_bounds__\s*").match(text, i)
            if b:
                i = closing(text, b.end(), "()") + 1
            k = re.compile(r"[\s\w]*?(\w+)\s*\(").match(text, i)
            if not k:
                continue
            p1 = closing(text, k.end() - 1, "()")
            b0 = text.index("{", p1)
            yield os.path.basename(path), k.group(1), text[k.end():p1], text[b0 + 1:closing(text, b0, "{}")]


OVERLAPPED = [k for k in kernels() if "grid_wait()" in k[3]]


def test_the_overlapped_kernels_are_found():
    assert {(f, n) for f, n, _, _ in OVERLAPPED} == {
        ("small.cuh", "k_force"), ("small.cuh", "k_force_ahead"), ("small.cuh", "k_force_sums"),
        ("small.cuh", "k_force_occ"), ("split.cuh", "k_force"), ("mma64.cuh", "k_link")}


@pytest.mark.parametrize("file,name,params,body", OVERLAPPED, ids=[f"{f}:{n}" for f, n, _, _ in OVERLAPPED])
def test_waits_first_and_promises_nothing_about_fields(file, name, params, body):
    assert body.strip().startswith("grid_wait();")
    for p in params.split(","):
        # the job table and its list of items are constant; everything else may be written by the launch before
        if not re.search(r"\b(table|items)$", p.strip()):
            assert "__restrict__" not in p, p


@pytest.mark.parametrize("file", ["common.cuh", "small.cuh", "split.cuh", "mma64.cuh"])
def test_fields_are_loaded_coherently_behind_the_wait(file):
    text = source(os.path.join(CSRC, file))
    assert "ld.global.nc" not in text and "ld.nc" not in text
    for m in re.finditer(r"__ldg\(", text):
        arg = text[m.end():closing(text, m.end() - 1, "()")]
        assert re.match(r"\s*(L\.nbr|nbr|items)\b", arg), arg
    for m in re.finditer(r"\basm\b(\s+volatile)?\s*\(", text):
        if "ld.global" in text[m.end():closing(text, m.end() - 1, "()")]:
            assert m.group(1), text[m.start():m.start() + 80]
