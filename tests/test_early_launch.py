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


def test_a_kernel_lets_its_dependents_in_when_it_holds_its_tmem():
    """A dependent that took the SM's TMEM first would wait for this kernel, and this kernel for the TMEM."""
    kernels = [k for path in SOURCES for k in _code(path).split("__global__")[1:] if "tmem_alloc" in k]
    kernels = [k.split("\n}\n")[0] for k in kernels]
    kernels = [k for k in kernels if re.search(r"\btmem_alloc2?\(", k)]
    assert len(kernels) == 6
    for k in kernels:
        assert re.findall(r"\b(tmem_alloc|tmem_relinquish|pdl_trigger|pdl_wait)2?\(", k) == [
            "tmem_alloc", "tmem_relinquish", "pdl_trigger", "pdl_wait"], k[:200]


def test_the_sources_are_there():
    assert len(SOURCES) > 20
