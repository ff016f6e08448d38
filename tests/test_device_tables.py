"""Declarations of the device tables that the CUDA sources read as structs."""
import glob
import os
import re

from conftest import ROOT


def test_constant_tables_have_their_elements_alignment():
    """A __constant__ char array has alignment 1: read as a struct of pointers
    and 64-bit strides its address must be declared aligned, or the array
    declared as what it holds."""
    seen = 0
    for path in sorted(glob.glob(os.path.join(ROOT, "pywave_b200", "csrc", "*.cu*"))):
        with open(path) as f:
            text = f.read()
        for decl in re.findall(r"^\s*(?:static\s+)?__constant__[^;]*;", text, re.M):
            seen += 1
            assert "char" not in decl or "__align__" in decl, f"{os.path.basename(path)}: {decl}"
    assert seen >= 1
