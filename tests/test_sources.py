"""Rules of the device sources that no run can show reliably."""
import glob
import os
import re

import pytest

from helpers import ROOT

SRC = os.path.join(ROOT, "tval3-cpu_b200", "csrc")


@pytest.mark.parametrize("name", ["ops.cu", "unroll.cu", "kernels.cu"])
def test_vectors_are_not_read_as_constants(name):
    """Kernels launched as programmatic dependents are resident while the kernel before them still writes their input
    vector: x and y (and the unrolled solve's R.x) go through ld_vec, never through __ldg or another ld.global.nc."""
    with open(os.path.join(SRC, name)) as f:
        code = re.sub(r"//[^\n]*", "", f.read())
    reads = [r.strip() for r in re.findall(r"__ldg\(([^;]*)", code)]
    vectors = [r for r in reads if re.match(r"(?:[xyp]|R\.x)\s*(?:\)|\+)", r)]
    assert not vectors, vectors


def test_sources_are_there():
    assert len(glob.glob(os.path.join(SRC, "*.cu"))) >= 9
