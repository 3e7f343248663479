"""Meshes other than ordinary triangles: cells of four to six and more neighbours, which leave the
unrolled forms of the slopes and of their reverse, and centroids whose distances div_known may not
divide by (slope_component_ok).  The run kernel, the step's kernels and the oracle give the same bits,
and the gradient is that of the replayed cost."""
import numpy as np
import pytest

from oracle import binding
from tests.conftest import load_pkg

pytestmark = pytest.mark.gpu


def merged_mesh(pkg, nx, ny, lx, ly, width, seed=1, z_fn=None):
    """The cells of a jittered grid of quads, `width` quads in a row merged into one cell (odd rows half
    a cell off, as bricks are laid): up to 2 width + 2 neighbours."""
    from dataclasses import replace

    m = pkg.mesh.jittered_triangle_mesh(nx, ny, lx, ly, seed=seed, z_fn=z_fn)
    q = np.arange(m.cell_nb) // 2
    row, col = q // nx, q % nx
    label = row * (nx + 2) + (col + (row % 2) * (width // 2)) // width
    group = np.unique(label, return_inverse=True)[1]
    n = int(group.max()) + 1
    area = np.bincount(group, m.cell_area, n)

    def mean(v):
        return np.bincount(group, v * m.cell_area, n) / area

    L, R = group[m.edge_int_cells[:, 0]], group[m.edge_int_cells[:, 1]]
    keep = np.nonzero(L != R)[0]
    flip = np.where(L[keep] > R[keep], -1.0, 1.0)
    lo, hi = np.minimum(L[keep], R[keep]), np.maximum(L[keep], R[keep])
    o = np.lexsort((hi, lo))
    keep, flip, lo, hi = keep[o], flip[o], lo[o], hi[o]
    bo = np.argsort(group[m.edge_bnd_cell], kind="stable")
    e = {k: getattr(m, f"edge_int_{k}")[keep] for k in ("nodes", "length", "mx", "my", "mz", "dnorm")}
    b = {k: getattr(m, f"edge_bnd_{k}")[bo] for k in ("nodes", "length", "nx", "ny", "mx", "my", "mz", "dnorm", "code")}
    return replace(m, cell_nodes=[], cell_nodes_flat=None, cell_area=area, cell_perimeter=np.zeros(n), cell_x=mean(m.cell_x),
                   cell_y=mean(m.cell_y), cell_z_b=mean(m.cell_z_b), edge_int_cells=np.stack([lo, hi], 1).astype(np.int64),
                   edge_int_nx=m.edge_int_nx[keep] * flip, edge_int_ny=m.edge_int_ny[keep] * flip,
                   edge_bnd_cell=group[m.edge_bnd_cell][bo].astype(np.int64),
                   **{f"edge_int_{k}": v for k, v in e.items()}, **{f"edge_bnd_{k}": v for k, v in b.items()})


def degrees(mesh):
    return np.bincount(mesh.edge_int_cells.reshape(-1), minlength=mesh.cell_nb)


def _case(pkg, mesh, scheme="muscl_evr"):
    rng = np.random.default_rng(mesh.cell_nb)
    n = mesh.cell_nb
    h0 = np.maximum(0.0, 1.0 + 0.3 * np.sin(0.5 * mesh.cell_x) - mesh.cell_z_b)
    opts = {"model_hyperb": "sp", "model_friction": "manning", "num_scheme": scheme, "topo_discretization": "discontinuous",
            "cfl_max": 0.7, "dt_max": 10.0, "dt_map": 100.0, "h_min": 1e-5, "t_max": 1.0e6, "store_flag": "none",
            "output_format": "txt"}
    return pkg.case.Case(mesh=mesh, opts=opts, h0=h0, q0=0.2 * h0 * rng.uniform(-1, 1, n), r0=0.2 * h0 * rng.uniform(-1, 1, n),
                         phi=rng.uniform(0.6, 1.0, n), boussinesq=np.ones(n), friction=np.stack([np.full(n, 0.03)] * 2 + [np.zeros(n)]),
                         bc=pkg.workloads._wall_series(mesh.bc_codes()), extra={})


def _bed(x, y):
    return 0.9 * np.exp(-((x - 8.0) ** 2 + (y - 5.0) ** 2) / 6.0)


def _bits(a):
    return np.ascontiguousarray(a, dtype=np.float64).view(np.int64)


def _forms_agree(pkg, case, calls=(1, 40, 9)):
    binding.build(reference=False)
    oracle = binding.SpOracle(case, portable_math=True)
    models = []
    for run in (1, 0):
        m = pkg.SpModel(case)
        m.set_option("run_kernel", run)
        models.append(m)
    for n in calls:
        oracle.step(n)
        for m in models:
            assert m.step(n) == n
            assert all(np.array_equal(_bits(x), _bits(y)) for x, y in zip(m.state(), oracle.state()))
    for name in ("slope_x", "slope_y"):
        assert np.array_equal(_bits(models[0].array(name)), _bits(models[1].array(name)))
    for m in models:
        m.close()


# width 1: quads (4 neighbours); 2: bricks (6); 4: 8 to 10 neighbours.  About 300 cells (a pair of lanes per
# slope) and 27,000 (a lane per slope)
@pytest.mark.parametrize("width,most", [(1, 4), (2, 6), (4, 10)])
@pytest.mark.parametrize("quads", [(24 * 1, 12), (240, 112)])
def test_many_neighbours(width, most, quads):
    pkg = load_pkg()
    mesh = merged_mesh(pkg, quads[0] * width, quads[1], 24.0, 10.0, width, z_fn=_bed)
    d = degrees(mesh)
    assert d.max() == most
    _forms_agree(pkg, _case(pkg, mesh), calls=(1, 40, 9) if quads[0] < 100 else (1, 6))


def _odd_mesh(pkg, y):
    """Triangles; an interior cell's centroid at y = 0 and a neighbour's at `y`."""
    m = pkg.mesh.jittered_triangle_mesh(24, 12, 24.0, 10.0, seed=2, z_fn=_bed)
    lo, hi = m.edge_int_cells[m.edge_int_nb // 2]
    shift = m.cell_y[lo]
    m.cell_y, m.edge_int_my, m.edge_bnd_my = m.cell_y - shift, m.edge_int_my - shift, m.edge_bnd_my - shift
    m.cell_y[hi] = y
    return m


@pytest.mark.parametrize("y", [0.0, 1e-70])     # 1e-70: the slopes of the whole mesh divide in full
def test_lengths_out_of_range(y):
    pkg = load_pkg()
    _forms_agree(pkg, _case(pkg, _odd_mesh(pkg, y)))


def _gradient_error(pkg, case, rng):
    """|adjoint - central difference| / |adjoint| of the cost by h0, along a smooth direction"""
    m = pkg.SpModel(case)
    n = m.record(12, 5)
    cells = np.arange(0, m.n, 7)
    m.set_observations(cells, [6, n], np.tile(case.h0[cells] * 1.1, (2, 1)))
    g = m.adjoint()[1]
    d = case.h0 * np.sin(0.3 * case.mesh.cell_x + rng.uniform(0, 6))
    J = []
    eps = 1e-6
    for s in (1.0, -1.0):
        m.set_trajectory_start(case.h0 + s * eps * d, case.q0, case.r0)
        J.append(m.replay_cost())
    m.close()
    ad = float(g["h0"] @ d)
    return abs(ad - (J[0] - J[1]) / (2 * eps)) / abs(ad), g


# a wet bed without fronts, so that no branch lies within the difference's step
@pytest.mark.parametrize("width", [1, 2])
def test_gradient_with_many_neighbours(width):
    pkg = load_pkg()
    rng = np.random.default_rng(width)
    case = _case(pkg, merged_mesh(pkg, 24 * width, 12, 24.0, 10.0, width))
    assert min(_gradient_error(pkg, case, rng)[0] for _ in range(3)) < 1e-5


def test_gradient_with_lengths_out_of_range():
    pkg = load_pkg()
    got = [_gradient_error(pkg, _case(pkg, _odd_mesh(pkg, y)), np.random.default_rng(1)) for y in (0.0, 1e-70)]
    assert got[0][0] < 1e-5 and got[1][0] < 1e-5
    for name in got[0][1]:
        a, b = (x[1][name] for x in got)
        assert np.max(np.abs(a - b)) <= 1e-12 * np.max(np.abs(a)), name
