"""Every kernel of a force pass waits for the kernels ahead of it before it
reads anything.

A pass kernel may be launched with programmatic stream serialization, and the
writes of the kernels ahead are visible only to threads past
griddepcontrol.wait.  The order is a property of the source, so it is read
there: in each kernel that launch_early or launch_pass starts, pass_kernel_entry
is the first statement, and no kernel body called from it waits by itself."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "dem3d_b200",
                    "csrc")
FILES = ("dem_lib.cu", "dem_kernels.cuh", "dem_mixed.cu", "dem_pass.cuh", "dem_test.cuh")


def _source():
    text = "".join(open(os.path.join(CSRC, f)).read() for f in FILES)
    return re.sub(r"//[^\n]*", "", text)


def _started_early(text):
    names = re.findall(r"launch_early\(\s*c,[^;]*?,\s*(k_\w+)", text)
    names += re.findall(r"launch_pass\(\s*early,\s*(k_\w+)", text)
    return sorted(set(names))


def test_the_pass_kernels_are_found():
    assert set(_started_early(_source())) >= {"k_relink", "k_rows", "k_lists", "k_test",
                                              "k_pair_fp64", "k_fold_fp64", "k_pair_mixed",
                                              "k_fold_mixed"}


@pytest.mark.parametrize("name", _started_early(_source()))
def test_a_pass_kernel_waits_first(name):
    found = re.findall(r"__global__[^;{]*?\b%s\([^{]*\{\s*([^;]*);" % name, _source())
    assert len(found) == 1
    assert found[0].strip() == "pass_kernel_entry()"


def test_nothing_else_waits():
    text = _source()
    assert text.count("griddepcontrol.wait") == 1
    assert text.count("pass_kernel_entry();") == len(_started_early(text))
