"""Node types declare the alignment that their 32-byte loads need."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.parametrize("node", ["GpuNode4", "QNode4", "HNode4"])
def test_nodes_are_32_byte_aligned(node):
    src = f'#include "bvh_build.h"\nstatic_assert(alignof(rtb200::{node}) % 32 == 0, "");\n'
    subprocess.run(["g++", "-std=c++17", "-fsyntax-only", "-I", os.path.join(ROOT, "rise_b200", "csrc"), "-x", "c++", "-"],
                   input=src, text=True, check=True)
