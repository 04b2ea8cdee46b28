"""Kernels that are launched with a programmatic dependency are resident while
the kernel before them still writes: what they read of it must not go through
non-coherent loads (ld.global.nc, __ldg), which are for data that is read-only
for a kernel's lifetime.  Checked in the source: no such load in a function
that waits for the previous kernel, nor in the row and factor loads that these
functions share."""
import glob
import os
import re

import pytest

from conftest import ROOT

CSRC = os.path.join(ROOT, "phist_b200", "csrc")
NC = re.compile(r"__ldg\s*\(|ld\.global\.nc|ld\.global\.L1::\w+\.nc")


def _bodies(text):
    return re.findall(r"^\{\n(.*?)^\}", text, re.S | re.M)


@pytest.mark.parametrize("path", sorted(glob.glob(os.path.join(CSRC, "*.cu*"))), ids=os.path.basename)
def test_no_noncoherent_loads_after_the_wait(path):
    for body in _bodies(open(path).read()):
        if "pdl_wait()" in body or "griddepcontrol.wait" in body:
            assert not NC.search(body)


@pytest.mark.parametrize("name", ["pb_spmmv_pf.cuh", "pb_spmmv_lz.cuh", "pb_krylov.cuh", "pb_frag.cuh", "pb_prec.cuh"])
def test_no_noncoherent_loads_in_the_files_of_these_kernels(name):
    assert not NC.search(open(os.path.join(CSRC, name)).read())


def test_shared_row_and_factor_loads():
    text = open(os.path.join(CSRC, "pb_spmmv.cuh")).read()
    head = text[:text.index("constexpr int SPMV_BS")]  # Vec, spmv_cscale
    assert "struct Vec" in head and "spmv_cscale" in head and not NC.search(head)
