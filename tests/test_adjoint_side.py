"""The reverse of the HLLC flux takes the tangential velocity's derivative on the side whose velocity the
forward took, down to the last bit of the discharge at which the mass flux changes sign
(tests/adjoint_side_check.cpp, built with g++ from the same source as the kernels)."""
import os
import subprocess

import pytest

from tests.test_adjoint_host import CSRC, ROOT, _compiler


@pytest.fixture(scope="module")
def results(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("side") / "adjoint_side_check")
    src = os.path.join(ROOT, "tests", "adjoint_side_check.cpp")
    subprocess.run([_compiler(), "-O2", "-std=c++17", "-ffp-contract=off", "-I", CSRC, src, "-o", exe], check=True,
                   capture_output=True)
    out = subprocess.run([exe], check=True, capture_output=True, text=True).stdout
    return {name: (int(n), int(differ)) for name, n, differ in (line.split() for line in out.splitlines())}


@pytest.mark.parametrize("topo", ["discontinuous", "blending"])
def test_the_forward_s_side(results, topo):
    n, differ = results[topo]
    assert n > 100000 and differ == 0
