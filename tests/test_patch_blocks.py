"""Blocks of the elementwise launches over a level's patches: enough for one large patch, never so
many that the idle ones of small patches cost more than the work."""
import os
import subprocess

import pytest

import configs  # noqa: F401  (puts the repository on the path)
from amrclaw_b200.build import CSRC, nvcc


@pytest.mark.parametrize("items,per,patches,blocks", [
    (1, 512, 1, 1), (512, 512, 1, 1), (513, 512, 1, 2), (4 * 1002 ** 2, 512, 1, 4096), (4 * 1000 ** 2, 512, 18, 1820),
    (4 * 56 ** 2, 512, 500, 25), (5 * 64 ** 3, 1024, 716, 45), (4 * 1000 ** 2, 512, 3000, 10), (10 ** 9, 512, 65535, 8), (64, 512, 65535, 1)])
def test_blocks(tmp_path, items, per, patches, blocks):
    src = tmp_path / "blocks.cpp"
    src.write_text('#include "common.cuh"\nstatic_assert(amrb::patch_blocks(%d, %d, %d) == %d, "");\n' % (items, per, patches, blocks))
    cuda = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(nvcc()))), "include")
    subprocess.run(["g++", "-std=c++17", "-fsyntax-only", "-I", CSRC, "-I", cuda, str(src)], check=True)
