"""The run kernel of small meshes (csrc/sw2d_run.cu: all steps of a call in one launch, tiles kept in
shared memory) against the step's own kernels, bit for bit: states, slopes, time, dt and the balance
slots that edges left dry keep, at meshes around a tile and around the pairs' and the whole form's
ranges, for every scheme, model, friction law and source."""
import numpy as np
import pytest

from tests.conftest import load_pkg

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def pkg():
    p = load_pkg()
    p.build.build()
    return p


def _bits(a):
    return np.ascontiguousarray(a, dtype=np.float64).view(np.int64)


def _walk(pkg, case, run, calls=(1, 2, 30, 0, 7)):
    """States after each of the calls, then after the same steps by the step kernels (which read the
    slots the run left)."""
    m = pkg.SpModel(case)
    m.set_option("run_kernel", run)
    out = []
    for n in calls:
        out.append((m.step(n), m.t, m.dt))
        out += [_bits(v) for v in m.state()]
    if str(case.opts["num_scheme"]) == "muscl_evr":
        out += [_bits(m.array("slope_x")), _bits(m.array("slope_y"))]
    m.set_option("run_kernel", 0)
    out.append((m.step(3), m.t, m.dt))
    out += [_bits(v) for v in m.state()]
    m.close()
    return out


def _same(pkg, case, **kw):
    a, b = _walk(pkg, case, 1, **kw), _walk(pkg, case, 0, **kw)
    for x, y in zip(a, b):
        assert x == y if isinstance(x, tuple) else np.array_equal(x, y)


@pytest.mark.parametrize("cells", [8, 60, 66, 130, 500, 5000, 19000, 24000])
@pytest.mark.parametrize("scheme", ["muscl_evr", "godunov"])
def test_mesh_sizes(pkg, cells, scheme):
    case = pkg.workloads.dam_break(n_cells=cells, scheme=scheme, mesh="delaunay" if cells < 10000 else "grid")
    rng = np.random.default_rng(cells)
    case.q0 = 0.2 * case.h0 * rng.uniform(-1, 1, case.mesh.cell_nb)
    _same(pkg, case, calls=(1, 2, 12))


@pytest.mark.parametrize("cells", [58000, 64000, 70000])
def test_largest_meshes(pkg, cells):
    _same(pkg, pkg.workloads.gaussian_bumps(n_cells=cells, initial="dam"), calls=(1, 5))


@pytest.mark.parametrize("friction", ["none", "chezy", "manning", "strickler"])
@pytest.mark.parametrize("scheme,topo", [("godunov", "blending"), ("muscl_evr", "discontinuous"), ("muscl_evr", "blending")])
def test_sources_and_topographies(pkg, friction, scheme, topo):
    for outflow, loss, b in (("fr", True, 1.0), ("h", False, 1.1), ("z", True, 1.0), ("q", False, 1.0)):
        case = pkg.workloads.channel_features(n_cells=900, scheme=scheme, topo=topo, friction=friction, outflow=outflow,
                                              head_loss=loss, boussinesq=b)
        _same(pkg, case, calls=(1, 60, 200))


@pytest.mark.parametrize("scheme,topo", [("godunov", "discontinuous"), ("godunov", "blending"),
                                         ("muscl_evr", "discontinuous"), ("muscl_evr", "blending")])
def test_dip(pkg, scheme, topo):
    for inflow, dissipation in (("q", True), ("phiWq", False)):
        case = pkg.workloads.dip_channel(n_cells=1500, scheme=scheme, topo=topo, inflow=inflow, dissipation=dissipation)
        _same(pkg, case, calls=(1, 60, 100))


def test_end_time_storage_times_and_long_calls(pkg):
    case = pkg.workloads.dam_break(n_cells=300, t_max=2.0)
    case.opts["dt_map"] = 0.25                      # snapped steps on the way
    ends = []
    for run in (1, 0):
        m = pkg.SpModel(case)
        m.set_option("run_kernel", run)
        done = [m.step(10), m.execute(), m.step(5)]  # the end inside a launch; nothing left after it
        m.set_t_max(400.0)
        done.append(m.step(2500))                    # more than one launch
        ends.append((done, m.t, m.dt, [_bits(v) for v in m.state()]))
        m.close()
    a, b = ends
    assert a[:3] == b[:3] and a[0][2] == 0 and a[0][3] == 2500
    assert all(np.array_equal(x, y) for x, y in zip(a[3], b[3]))


def test_states_set_from_outside_and_saved_points(pkg):
    case = pkg.workloads.channel_features(n_cells=1200)
    res = []
    for run in (1, 0):
        m = pkg.SpModel(case)
        m.set_option("run_kernel", run)
        m.step(40)
        m.save_point()
        m.step(17)
        h, q, r = m.state()
        m.restore_point()
        m.step(17)
        assert all(np.array_equal(_bits(x), _bits(y)) for x, y in zip((h, q, r), m.state()))
        m.set_state(h[::-1].copy() * 0 + 0.3, q, r)
        m.set_time(3.0, 0.01)
        m.step(25)
        m.set_option("record_fluxes", 1)             # recorded: the step's kernels take over
        m.step(2)
        res.append([_bits(v) for v in m.state()] + [_bits(m.array("F1_int"))])
        m.set_option("record_fluxes", 0)
        m.step(4)
        res[-1] += [_bits(v) for v in m.state()]
        m.close()
    assert all(np.array_equal(x, y) for x, y in zip(*res))


def test_errors_are_those_of_the_step(pkg):
    case = pkg.workloads.channel_features(n_cells=600, topo="discontinuous", impervious=True)
    codes = []
    for run in (1, 0):
        m = pkg.SpModel(case)
        m.set_option("run_kernel", run)
        with pytest.raises(pkg.Sw2dError) as e:
            m.step(50)
        codes.append(e.value.code)
        m.close()
    assert codes[0] == codes[1]


def test_wait_that_runs_out(pkg):
    """A poll limit of 0: a tile that does not find its neighbours' words at the first look gives up,
    every other one ends at its own limit, and the call reports it.  From the saved point, with the
    default limit again, the model runs as before."""
    m = pkg.SpModel(pkg.workloads.dam_break(n_cells=4000))
    m.save_point()
    m.step(20)
    end = [_bits(v) for v in m.state()]
    m.restore_point()
    m.set_option("run_wait_polls", 0)
    with pytest.raises(pkg.Sw2dError, match="run kernel ran out"):
        m.step(20)
    m.set_option("run_wait_polls", -1)
    m.restore_point()
    m.step(20)
    assert all(np.array_equal(x, _bits(y)) for x, y in zip(end, m.state()))
    m.close()
