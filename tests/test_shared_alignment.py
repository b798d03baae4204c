"""Shared memory that the kernels read or write 16 bytes at a time is declared on a
16-byte boundary: a float array alone promises 4, and where the compiler puts it then
depends on what else the kernel keeps there.  Checked on the sources: nothing runs."""
import glob
import os
import re

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SOURCES = sorted(glob.glob(os.path.join(ROOT, "distembed_gb300", "csrc", "*.cu")))
DECLARED = re.compile(r"__shared__\s+(?:__align__\((\d+)\)\s+)?[\w:]+\s+(\w+)\s*\[")
# the accesses of 16 bytes: row helpers, vector pointers, asynchronous copies
WIDE = (r"\b(?:load|store)_lanes<[^;]*?\(\s*\w+\s*,\s*{0}\b", r"reinterpret_cast<(?:const )?(?:float4|uint4|int4|double2) \*>\(\s*&?{0}\b",
        r"\b(?:bulk_g2s|cp_async16)\(\s*(?:dev::)?smem_u32\(\s*&?{0}\b")


def declarations(text):
    """(name, declared alignment, text of the kernel after the declaration) of each array."""
    for m in DECLARED.finditer(text):
        end = text.find("\n}\n", m.end())
        yield m.group(2), int(m.group(1) or 0), text[m.end():end]


@pytest.mark.parametrize("path", SOURCES, ids=[os.path.basename(p) for p in SOURCES])
def test_wide_accesses_have_aligned_shared_arrays(path):
    text = re.sub(r"//[^\n]*", "", open(path).read())
    for name, align, body in declarations(text):
        if any(re.search(w.format(re.escape(name)), body, re.S) for w in WIDE):
            assert align >= 16, f"{os.path.basename(path)}: {name} is accessed 16 bytes at a time"


def test_the_check_sees_the_arrays_it_is_about():
    text = open(os.path.join(ROOT, "distembed_gb300", "csrc", "de_plain.cu")).read()
    wide = {name for name, _, body in declarations(re.sub(r"//[^\n]*", "", text))
            if any(re.search(w.format(name), body, re.S) for w in WIDE)}
    assert {"negsm", "s_acc"} <= wide
