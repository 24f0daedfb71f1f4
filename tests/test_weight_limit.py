"""The default weight limit (1.5 * total weight / threshold) at the ends of the int
range, as the host compiles it: the device's conversion stops there."""
import os
import shutil
import subprocess

import pytest

from conftest import ROOT

PROGRAM = r"""
#include <cstdio>
#include <cstdlib>
#include "cm_internal.h"
int main(int argc, char **argv) {
  volatile long long t = atoll(argv[1]);
  volatile int c = atoi(argv[2]);
  printf("%d\n", (int)cm_weight_limit(t, c));
}
"""


@pytest.fixture(scope="module")
def limit(tmp_path_factory):
    if not shutil.which("g++"):
        pytest.skip("no g++")
    d = tmp_path_factory.mktemp("limit")
    (d / "limit.cpp").write_text(PROGRAM)
    exe = str(d / "limit")
    subprocess.check_call(["g++", "-std=c++17", "-O2", "-I", os.path.join(ROOT, "cumetis_gb300", "csrc"),
                           str(d / "limit.cpp"), "-o", exe])
    return lambda tvwgt, to: int(subprocess.check_output([exe, str(tvwgt), str(to)]))


@pytest.mark.parametrize("tvwgt,to,want", [
    (4761, 100, 71), (0, 5, 0), (1, 2, 0), (3, 1, 4),
    (1431655764, 1, 2147483646), (1431655765, 1, 2147483647), (1431655766, 1, 2147483647),
    (2**31 - 1, 1, 2147483647), (1 << 40, 1, 2147483647), (1 << 40, 1 << 20, 1572864), (1 << 62, 3, 2147483647),
    (-2, 1, -3), (-(1 << 40), 1, -2147483648)])
def test_weight_limit(limit, tvwgt, to, want):
    assert limit(tvwgt, to) == want
