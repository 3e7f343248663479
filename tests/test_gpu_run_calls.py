"""The run kernel (csrc/sw2d_run.cu) at the calls around it: meshes that its tiles hardly describe,
memory that it does not get, other handles in other threads, a model's first calls and the autotuner.
Whatever form takes the steps, they are taken, with the same bits."""
import numpy as np
import pytest

from oracle import binding
from tests.conftest import load_pkg

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def pkg():
    p = load_pkg()
    p.build.build()
    binding.build(reference=False)
    return p


def _bits(a):
    return np.ascontiguousarray(a, dtype=np.float64).view(np.int64)


def _same_state(a, b):
    return all(np.array_equal(_bits(x), _bits(y)) for x, y in zip(a.state(), b.state()))


def _separate_cells(pkg, n, scheme, friction):
    """n triangles that share no edge: no internal edge at all"""
    x = np.concatenate([[2.0 * i, 2.0 * i + 1.0, 2.0 * i + 0.3] for i in range(n)])
    y = np.tile([0.0, 0.1, 1.0], n)
    mesh = pkg.mesh.mesh_from_triangles(x, y, np.zeros(3 * n), np.arange(3 * n).reshape(n, 3))
    case = pkg.workloads.dam_break(n_cells=8, scheme=scheme, friction=friction)
    case.mesh = mesh
    case.h0, case.q0, case.r0 = np.linspace(0.5, 1.0, n), np.full(n, 0.2), np.full(n, -0.1)
    case.phi, case.boussinesq = np.full(n, 0.8), np.ones(n)
    case.friction = None if friction == "none" else np.stack([np.full(n, 0.03)] * 2 + [np.zeros(n)])
    case.bc = pkg.workloads._wall_series(mesh.bc_codes())
    return case


@pytest.mark.parametrize("n", [1, 3, 200])
@pytest.mark.parametrize("scheme", ["muscl_evr", "godunov"])
@pytest.mark.parametrize("friction", ["none", "manning"])
def test_cells_without_internal_edges(pkg, n, scheme, friction):
    case = _separate_cells(pkg, n, scheme, friction)
    a, b = pkg.SpModel(case), pkg.SpModel(case)
    a.set_option("run_kernel", 1)
    b.set_option("run_kernel", 0)
    oracle = binding.SpOracle(case, portable_math=True)
    for k in (1, 7, 40):
        assert a.step(k) == b.step(k) == oracle.step(k) == k
        assert _same_state(a, oracle) and _same_state(b, oracle) and a.time == b.time
    a.close()
    b.close()
