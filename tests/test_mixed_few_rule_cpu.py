"""Which mixed TaylorF2 batches spread their bins over the lanes (``mixed_few``): the
faster of the two launches, where the measurements show one to be faster by a tenth."""
import os
import shutil
import subprocess

import pytest

from bilby_gb300 import _build
from tests.conftest import ROOT

PROBE = r"""
#include <cstdio>
#include <cstdlib>
#include "gwl_internal.h"
int main(int, char** v) {
  std::printf("%d", (int)gwl::mixed_few(std::atoll(v[1]), std::atoll(v[2]), std::atoi(v[3]), std::atof(v[4])));
}
"""

# (duration, chunks of 512 bins from 20 Hz, detectors, points, few points' launch / the other one, us)
MEASURED = [
    (128.0, 508, 1, 72, 113, 172), (128.0, 508, 1, 217, 233, 187), (128.0, 508, 1, 290, 294, 196),
    (128.0, 508, 2, 72, 147, 207), (128.0, 508, 2, 201, 303, 231), (128.0, 508, 3, 72, 181, 238),
    (128.0, 508, 3, 201, 394, 318), (128.0, 252, 1, 146, 122, 174), (128.0, 252, 1, 438, 271, 184),
    (128.0, 252, 2, 146, 162, 211), (128.0, 252, 2, 292, 273, 220), (256.0, 503, 1, 73, 125, 146),
    (256.0, 503, 1, 146, 196, 159), (256.0, 503, 2, 36, 111, 170), (256.0, 503, 2, 146, 273, 196),
    (256.0, 503, 3, 48, 157, 204), (256.0, 503, 3, 97, 254, 217), (64.0, 254, 1, 290, 162, 211),
    (64.0, 254, 1, 580, 272, 222), (64.0, 254, 2, 217, 173, 244), (64.0, 254, 2, 604, 383, 270),
    (64.0, 126, 1, 292, 131, 218), (64.0, 126, 1, 877, 294, 229), (64.0, 126, 3, 292, 212, 302),
    (48.0, 95, 1, 776, 205, 232), (48.0, 95, 1, 1552, 370, 242), (48.0, 95, 2, 582, 212, 267),
    (32.0, 127, 1, 1161, 270, 382), (32.0, 63, 2, 1170, 268, 470), (16.0, 64, 1, 2304, 232, 262),
    (8.0, 32, 1, 4608, 130, 221), (8.0, 16, 3, 3072, 127, 238), (8.0, 16, 2, 288, 55, 250),
    (4.0, 8, 1, 18432, 291, 358), (4.0, 8, 2, 9216, 183, 268), (4.0, 4, 2, 18432, 302, 387)]


@pytest.fixture(scope="module")
def rule(tmp_path_factory):
    gxx = shutil.which("g++")
    cuda = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(_build.nvcc()))), "include")
    if gxx is None or not os.path.isdir(cuda):
        pytest.skip("no host compiler or CUDA headers")
    tmp = tmp_path_factory.mktemp("rule")
    (tmp / "probe.cpp").write_text(PROBE)
    exe = tmp / "probe"
    subprocess.run([gxx, "-std=c++17", "-w", "-I", os.path.join(ROOT, "bilby_gb300", "csrc"), "-I",
                    os.path.join(ROOT, "include"), "-I", cuda, str(tmp / "probe.cpp"), "-o", str(exe)], check=True)
    return lambda *q: subprocess.run([str(exe), *map(str, q)], capture_output=True, text=True, check=True).stdout == "1"


@pytest.mark.parametrize("case", MEASURED)
def test_the_faster_launch(rule, case):
    duration, chunks, detectors, points, few, other = case
    assert rule(points, chunks, detectors, duration) == (few < other)


def test_limits_of_the_grid(rule):
    assert rule(65535, 1, 1, 2.0) and not rule(65536, 1, 1, 2.0)
    assert rule(1, 508, 3, 128.0) and rule(1, 147456, 1, 4.0) and not rule(1, 147457, 1, 4.0)
