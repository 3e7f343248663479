"""The gradient of a cell does not depend on which cells share its warp.

Narrow basins on one mesh, A and B in turn, with dry ridges several cells wide between them that
neither overtops, and a time step that dt_max fixes: nothing that happens in B reaches A.  The cells
are numbered along a space-filling curve, so that many warps hold cells of both.  B's basins have
gauges of their own; their Boussinesq coefficient changes how their wave-speed roots are
differentiated (1: in closed form), and A's gradient has to keep its bits."""
import numpy as np
import pytest

from tests.conftest import load_pkg

pytestmark = pytest.mark.gpu

DT = 0.01


def _case(pkg, scheme, b_other):
    w = pkg.workloads
    mesh = pkg.mesh.jittered_triangle_mesh(72, 72, 72.0, 72.0, seed=3)
    side = (mesh.cell_x - mesh.cell_y) % 16.0
    a, other = side < 4.0, (side >= 8.0) & (side < 12.0)
    ridge = ~(a | other)
    near, (L, R) = a, mesh.edge_int_cells.T        # A and the cells within three edges of it
    for _ in range(3):
        more = near.copy()
        more[R[near[L]]] = True
        more[L[near[R]]] = True
        near = more
    assert not np.any(near & other)
    mesh.cell_z_b = np.where(ridge, 5.0, 0.0)
    rng = np.random.default_rng(5)
    n = mesh.cell_nb
    h0 = np.where(ridge, 0.0, 1.0 + 0.2 * np.sin(0.4 * mesh.cell_x) * np.cos(0.3 * mesh.cell_y))
    q0, r0 = (0.3 * h0 * rng.uniform(-1, 1, n) for _ in range(2))
    opts = {"model_hyperb": "sp", "model_friction": "none", "num_scheme": scheme, "topo_discretization": "discontinuous",
            "cfl_max": 0.9, "dt_max": DT, "dt_map": 100.0, "h_min": 1e-5, "t_max": 40 * DT, "store_flag": "none",
            "output_format": "txt"}
    case = pkg.case.Case(mesh=mesh, opts=opts, h0=h0, q0=q0, r0=r0, phi=rng.uniform(0.6, 1.0, n),
                         boussinesq=np.where(a | ridge, 1.0, b_other), friction=None, bc=w._wall_series(mesh.bc_codes()),
                         extra={})
    gauges = np.sort(np.concatenate([rng.choice(np.nonzero(a)[0], 300, replace=False),
                                     rng.choice(np.nonzero(other)[0], 300, replace=False)]))
    return case, a, other, gauges


def _mixed_warps(model, a, other):
    perm = model.cell_permutation()       # the caller's cell of each cell in the library's order
    k = a.size // 32 * 32
    return int(np.sum(a[perm][:k].reshape(-1, 32).any(1) & other[perm][:k].reshape(-1, 32).any(1)))


@pytest.mark.parametrize("scheme", ["muscl_evr", "godunov"])
def test_adjoint(scheme):
    pkg = load_pkg()
    out = []
    for b in (1.0, 1.1):
        case, a, other, gauges = _case(pkg, scheme, b)
        model = pkg.SpModel(case)
        n = model.record(30, 10)
        assert n == 30 and np.all(model.trajectory_dt() == DT) and _mixed_warps(model, a, other) > 60
        model.set_observations(gauges, [10, 20, 30], np.tile(case.h0[gauges] * 1.05, (3, 1)))
        g = model.adjoint()[1]
        assert np.count_nonzero(g["h0"][a]) > 2000 and np.count_nonzero(g["h0"][other]) > 2000
        out.append(g)
        model.close()
    for name in out[0]:
        assert np.array_equal(out[0][name][a].view(np.int64), out[1][name][a].view(np.int64)), name


@pytest.mark.parametrize("scheme", ["muscl_evr", "godunov"])
def test_porosity_gradient(scheme):
    pkg = load_pkg()
    out = []
    for b in (1.0, 1.1):
        case, a, other, gauges = _case(pkg, scheme, b)
        model = pkg.SpModel(case)
        model.assim_configure(phi_transform="none", cost_normalize=True)
        times = DT * np.array([10.0, 20.0, 30.0])
        model.assim_set_gauges(times, gauges, np.ones(gauges.size), np.tile(case.h0[gauges] * 1.05, (3, 1)))
        steps, _ = model.assim_record(case.phi, 10)
        dt = model.assim_steps()[0]
        g, info = model.assim_gradient(case.phi, 10)
        assert info["n_nonfinite"] == 0 and np.count_nonzero(g[a]) > 2000
        out.append((dt, g))
        model.close()
    assert np.array_equal(out[0][0], out[1][0])
    assert np.array_equal(out[0][1][a].view(np.int64), out[1][1][a].view(np.int64))
