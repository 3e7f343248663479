"""Adjoints near the end of the range spread no further through the slope limiter's reverse than with plain
divisions (tests/adjoint_overflow_check.cpp, built with g++ from the same source as the kernels)."""
import os
import subprocess

import pytest

from tests.test_adjoint_host import CSRC, ROOT, _compiler


@pytest.fixture(scope="module")
def results(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("overflow") / "adjoint_overflow_check")
    src = os.path.join(ROOT, "tests", "adjoint_overflow_check.cpp")
    subprocess.run([_compiler(), "-O2", "-std=c++17", "-ffp-contract=off", "-I", CSRC, src, "-o", exe], check=True,
                   capture_output=True)
    out = subprocess.run([exe], check=True, capture_output=True, text=True).stdout
    return {int(line.split()[0]): [int(v) for v in line.split()[1:]] for line in out.splitlines()}


@pytest.mark.parametrize("neighbours", range(2, 7))
def test_no_entry_is_lost(results, neighbours):
    entries, nonfinite, lost = results[neighbours]
    assert entries == 40000 * (neighbours + 1) and nonfinite > 0   # the range is reached
    assert lost == 0
