"""Kernel attributes belong to a device, not to the process.

A launch that needs more shared memory than the default sets the attribute
on every call or where its plan is made; a flag that sets it once a process
would leave the kernels of a second device without it.  There is one device
here, so the sources are read: no function that sets an attribute keeps a
static flag.
"""
import glob
import os
import re

import pytest

from conftest import ROOT

SOURCES = sorted(glob.glob(os.path.join(ROOT, "dennou-ccm_gb300", "csrc", "*.cu")))


def _functions(text):
    """Bodies of the definitions that start in the first column."""
    for m in re.finditer(r"^(?:template [^\n]*\n)?[a-z][^\n;]*\([^;{]*\{\n", text, re.M):
        end = text.find("\n}\n", m.end())
        yield text[m.start():end]


@pytest.mark.parametrize("path", SOURCES, ids=os.path.basename)
def test_no_attribute_once_a_process(path):
    for body in _functions(open(path).read()):
        if "cudaFuncSetAttribute" in body:
            assert not re.search(r"^\s+static\b", body, re.M), body[:80]


def test_functions_are_found():
    text = open(os.path.join(ROOT, "dennou-ccm_gb300", "csrc", "legendre_dg.cu")).read()
    assert any("cudaFuncSetAttribute" in b for b in _functions(text))
