"""The exact rules the step takes in place of general operations, against those operations: a
division by a divisor of known reciprocal (div_known), the root of the wave speeds at a Boussinesq
coefficient of 1 (root_is_c), and the slopes at level differences outside div_known's range."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from tests.conftest import ROOT, load_pkg

CSRC = os.path.join(ROOT, "inria-internship-project-sw2d-enzyme_b200", "csrc")

SRC = r"""
#include "sp_math.cuh"
using namespace sw2d;
extern "C" long known(const double* x, const double* d, long n) {
    long bad = 0;
    for (long i = 0; i < n; i++) {
        const double q = x[i] / d[i], k = div_known(x[i], d[i], 1.0 / d[i]);
        bad += sw2d_pm_bits(q) != sw2d_pm_bits(k);
    }
    return bad;
}
extern "C" int in_range(double x) { return div_range_ok(x); }
extern "C" long root(const double* u, const double* c, long n, long* taken) {
    long bad = 0;
    for (long i = 0; i < n; i++) {
        if (!root_is_c(1.0, u[i], c[i])) continue;
        ++*taken;
        bad += sw2d_pm_bits(std::sqrt((1.0 - 1.0) * 1.0 * u[i] * u[i] + c[i] * c[i])) != sw2d_pm_bits(c[i]);
    }
    return bad;
}
"""


@pytest.fixture(scope="module")
def rules(tmp_path_factory):
    d = tmp_path_factory.mktemp("rules")
    (d / "r.cpp").write_text(SRC)
    so = d / "r.so"
    subprocess.run(["g++", "-std=c++17", "-O2", "-fPIC", "-ffp-contract=off", "-shared", "-I", CSRC, "-o", str(so),
                    str(d / "r.cpp")], check=True)
    lib = ctypes.CDLL(str(so))
    lib.in_range.argtypes = [ctypes.c_double]
    lib.known.restype = lib.root.restype = ctypes.c_long
    return lib


def _p(a):
    return a.ctypes.data_as(ctypes.c_void_p)


@pytest.mark.parametrize("kind", ["uniform", "wide", "near_one", "zeros"])
def test_division_by_a_known_reciprocal_is_the_ieee_quotient(rules, kind):
    rng = np.random.default_rng(3)
    n = 1_000_000
    if kind == "uniform":
        x, d = rng.uniform(-2, 2, n), rng.uniform(1, 2, n)
    elif kind == "wide":   # level difference times component over length, then over length again
        x = rng.choice([-1.0, 1.0], n) * 10.0 ** rng.uniform(-210, 180, n)
        d = 10.0 ** rng.uniform(-30, 30, n)
    elif kind == "near_one":   # mantissas next to 1 and 2, where quotients lie next to a rounding boundary
        x = 1.0 + rng.integers(0, 4096, n) * 2.0 ** -52
        d = np.where(rng.random(n) < 0.5, 1.0 + rng.integers(0, 4096, n) * 2.0 ** -52,
                     2.0 - rng.integers(1, 4096, n) * 2.0 ** -52)
    else:
        x, d = np.where(rng.random(n) < 0.5, 0.0, -0.0), rng.uniform(1e-30, 1e30, n)
    x, d = np.ascontiguousarray(x), np.ascontiguousarray(d)
    assert rules.known(_p(x), _p(d), ctypes.c_long(n)) == 0


def test_range_of_level_differences(rules):
    for v in (0.0, -0.0, 2.0 ** -498, -2.0 ** -498, 1e-16, -3.0, 2.0 ** 497):
        assert rules.in_range(v)
    for v in (2.0 ** -499, 5e-324, 1e-310, 2.0 ** 498, np.inf, -np.inf, np.nan):
        assert not rules.in_range(v)


def test_root_of_the_wave_speeds_at_boussinesq_one(rules):
    rng = np.random.default_rng(4)
    n = 1_000_000
    c = np.concatenate([10.0 ** rng.uniform(-139, 149, n), rng.uniform(0, 20, n), [0.0, -0.0, 1e-141, 1e200, np.inf, np.nan]])
    u = np.concatenate([rng.choice([-1.0, 1.0], 2 * n) * 10.0 ** rng.uniform(-300, 299, 2 * n),
                        [-3.0, 1.0, 1.0, 1.0, 1.0, 1.0]])
    taken = ctypes.c_long(0)
    assert rules.root(_p(u), _p(c), ctypes.c_long(c.size), ctypes.byref(taken)) == 0
    assert taken.value == 2 * n + 1   # all but -0, 1e-141, 1e200, inf and NaN


@pytest.mark.gpu
@pytest.mark.parametrize("depth", [1e-200, 5e-324, 1e-16])
def test_slopes_where_level_differences_leave_the_range(depth):
    """A flat bed whose right part holds a film of `depth`: level differences down to the smallest
    double take the general division, cell by cell."""
    pkg = load_pkg()
    pkg.build.build()
    from oracle import binding
    binding.build(reference=False)
    case = pkg.workloads.dam_break(n_cells=700, mesh="delaunay")
    rng = np.random.default_rng(1)
    case.h0 = np.where(case.mesh.cell_x < 30.0, 1.0, np.where(rng.random(case.mesh.cell_nb) < 0.5, depth, 0.0))
    gpu, cpu = pkg.SpModel(case), binding.SpOracle(case, portable_math=True)
    for _ in range(3):
        gpu.step(1), cpu.step(1)
        for a, b in zip((gpu.array("slope_x"), gpu.array("slope_y")) + gpu.state(),
                        (cpu.array("slope_x"), cpu.array("slope_y")) + tuple(cpu.state())):
            assert np.array_equal(np.asarray(a).view(np.int64), np.asarray(b).view(np.int64))
    gpu.close()
