"""Vector accesses to shared memory: an array of scalars is only aligned to its
element, so one that is read or written several elements at a time says so in
its declaration.  Checked in the source: in every kernel, the static shared
arrays (and the pointers set to a place inside them) that reach a paired store,
a paired load or a cast to a vector type carry __align__(16) or are of a
vector type themselves."""
import glob
import os
import re

import pytest

from conftest import ROOT

FILES = sorted(glob.glob(os.path.join(ROOT, "phist_b200", "csrc", "*.cu*")))
DECL = re.compile(r"__shared__\s+((?:__align__\(\d+\)\s+)?)(double|float|T|int|unsigned char)\s+(\w+)\s*\[")
VECTOR = r"(?:frag_st2|frag_ld2|reinterpret_cast<(?:const )?(?:double|float|int)[24]\*>|Vec<[^>]*>::\w+)\s*\(\s*%s\b"


def _bodies(text):
    """the function bodies of a file (text between a { in column 0 and its })"""
    return re.findall(r"^\{\n(.*?)^\}", text, re.S | re.M)


def unaligned(text):
    bad = []
    for body in _bodies(text):
        for align, _, name in DECL.findall(body):
            names = {name}
            while True:
                more = {p for p, q in re.findall(r"\*\s*(\w+)\s*=\s*(?:reinterpret_cast<[^>]*>\()?\s*(\w+)", body)
                        if q in names}
                if more <= names:
                    break
                names |= more
            if not align and any(re.search(VECTOR % n, body) for n in names):
                bad.append(name)
    return bad


@pytest.mark.parametrize("path", FILES, ids=os.path.basename)
def test_vector_accesses_are_aligned(path):
    assert unaligned(open(path).read()) == []


def test_rule_sees_a_scalar_array():
    kernel = "{\n  __shared__ %sdouble sm[64];\n  double* tile = sm + 8;\n  frag_st2(tile + 2, 0.0, 0.0);\n}\n"
    assert unaligned(kernel % "") == ["sm"] and unaligned(kernel % "__align__(16) ") == []
