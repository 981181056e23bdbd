"""CPU check of how the stencil kernels stage a block (no GPU needed).

RBGS passes are programmatic dependents of one another: a pass is resident
while the one before it still writes the iterate and the pushed guides, which
the read-only load path does not allow for.  tests/native/staging_check.cpp
compiles the staging code for the host, counts the reads that take that path
and compares every staged value; the source of the dependent kernel is checked
to stage that way and to keep the path for what no pass writes."""
import os
import re
import subprocess

import pytest

import ffvgpu
from test_cpu_bounds import ROOT, table_text

SRC = os.path.join(ROOT, "tests", "native", "staging_check.cpp")
CSRC = os.path.join(ROOT, "ffv-hc_b200", "csrc")
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")


@pytest.fixture(scope="module")
def checker(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("staging") / "staging_check")
    subprocess.run(["g++", "-O1", "-std=c++17", "-w", "-I", os.path.join(CUDA, "include"),
                    "-o", exe, SRC], check=True)
    return exe


@pytest.mark.parametrize("level,kw", [(0, {}), (2, {}), (3, dict(center=(2.3, -1.1, 0.7), radius=0.8))])
def test_staged_blocks_and_their_read_path(checker, level, kw):
    g = ffvgpu.SphereGrid(level, **kw)
    out = subprocess.run([checker], input=table_text(g), capture_output=True, text=True, check=True)
    wrong, written, readonly = map(int, out.stdout.split())
    assert wrong == 0, "a staged value differs"
    assert written == 0, "x or guides of a dependent launch read through the read-only path"
    assert readonly > 0  # the count sees the reads it is meant to see


def test_dependent_kernels_read_what_passes_write_with_ordinary_loads():
    users = []
    for name in sorted(os.listdir(CSRC)):
        with open(os.path.join(CSRC, name)) as f:
            code = re.sub(r"//[^\n]*", "", f.read())
        if not name.endswith(".cu") or "launch_dep(" not in code:
            continue
        users.append(name)
        assert "ReadOnly" not in code and not re.search(r"const double\s*\*\s*__restrict__\s+(xin|gst)", code)
        assert set(re.findall(r"Staging<([^>]*)>", code)) <= {"SRC, Written"}, name
        assert set(re.findall(r"guide_pair(<\w+>)?\(", code)) <= {"<Written>"}, name
        assert set(re.findall(r"__ldg\(\s*(\w+)", code)) <= {"order", "C"}, name  # C: the uniform records
    assert users == ["rbgs_block.cu", "rbgs_ring.cu"]
