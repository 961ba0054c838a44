"""Every C++ header of the cuda device compiles as a translation unit's only
include: which headers a source lists, and in which order, must not decide
whether a build from nothing succeeds."""
import glob
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "openvkl_b200", "csrc")
HEADERS = sorted(os.path.basename(p) for p in glob.glob(os.path.join(CSRC, "*.h")))


@pytest.mark.parametrize("header", HEADERS)
def test_header_compiles_alone(header):
    from openvkl_b200 import build
    cuda = os.path.join(os.path.dirname(os.path.dirname(build.NVCC)), "include")
    r = subprocess.run(["g++", "-std=c++17", "-fsyntax-only", "-x", "c++", "-I", CSRC, "-I", cuda, "-"],
                       input=f'#include "{header}"\n', capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
