"""The largest graph that the kernel of whole levels may be built for: its packed
scans hold counts below 2^21, and a graph of that many isolated vertices has as many
coarse ones."""
import os
import shutil
import subprocess

import pytest

from cumetis_gb300 import build as B


@pytest.mark.skipif(not shutil.which("nvcc"), reason="no nvcc")
@pytest.mark.parametrize("work,fits", [(2097152, False), (2097151, True)])
def test_limit_is_checked_when_built(tmp_path, work, fits):
    src = os.path.join(B.CSRC, "cm_levels.cu")
    cmd = ["nvcc", "-std=c++17", *B.ARCH, "-I" + B.INCLUDE, "-DCM_FUSED_WORK=%d" % work, "-cuda", src, "-o",
           str(tmp_path / "levels.ii")]  # the front end only
    r = subprocess.run(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
    assert (r.returncode == 0) == fits, r.stdout[-2000:]
    assert fits or "packed scan" in r.stdout
