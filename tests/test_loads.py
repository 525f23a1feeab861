"""Kernels of the library start before the kernels ahead of them in the stream have ended. What those write is
not read-only while a kernel runs, so the non-coherent load path, for which the compiler may move a load above
the wait for them, is closed to all of them."""
import glob
import os
import re

import pytest

from conftest import ROOT

SOURCES = sorted(glob.glob(os.path.join(ROOT, "nanospeaker_b200", "csrc", "*.cu*")))


def _code(path):
    with open(path) as f:
        return re.sub(r"//[^\n]*", "", f.read())


@pytest.mark.parametrize("path", SOURCES, ids=os.path.basename)
def test_no_kernel_takes_the_non_coherent_load_path(path):
    assert not re.findall(r"\b__ldg\b|ld\.global\.nc|\b__restrict__", _code(path))


def test_the_sources_are_there():
    assert len(SOURCES) > 20
