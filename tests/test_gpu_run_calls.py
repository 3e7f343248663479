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


@pytest.mark.parametrize("scheme", ["muscl_evr", "godunov"])
def test_no_memory_for_the_tiles(pkg, scheme):
    """Each of the run kernel's allocations fails in turn: the step's kernels take the steps, no error
    stays behind, and the option set again tries again."""
    case = pkg.workloads.dam_break(n_cells=3000, scheme=scheme)
    want = pkg.SpModel(case)
    fails = want.lib.sw2d_test_fail_allocations
    fails(0, 0)
    want.set_option("run_kernel", 1)
    want.step(40)
    n = fails(0, 0)
    assert n > 0 and want.get_option("run_steps") == 40
    for skip in range(n):
        m = pkg.SpModel(case)
        m.set_option("run_kernel", 1)
        fails(skip, 1)
        try:
            assert m.step(40) == 40
        finally:
            fails(0, 0)
        assert m.get_option("run_steps") == 0 and _same_state(m, want) and m.time == want.time
        m.prepare()
        assert m.step(1) == 1 and m.get_option("run_steps") == 0
        m.set_option("run_kernel", 1)
        m.step(3)
        assert m.get_option("run_steps") == 3
        m.close()
    want.step(4)
    assert want.lib.sw2d_last_error(want.handle) == b""
    want.close()


def test_tiles_that_do_not_fit_hold_no_memory(pkg):
    """Under the size limit the tiles are built before their shared memory turns out too large (cells of
    six neighbours)."""
    import torch

    from tests.test_gpu_polygons import _case, merged_mesh

    case = _case(pkg, merged_mesh(pkg, 720, 170, 72.0, 34.0, 2))
    assert 60000 < case.mesh.cell_nb <= 66000
    m = pkg.SpModel(case)
    torch.cuda.synchronize()
    m.set_option("run_kernel", 1)
    m.set_option("run_kernel", 0)
    m.step(40)                       # graph and modules
    free0 = torch.cuda.mem_get_info(0)[0]
    m.set_option("run_kernel", 1)
    m.step(40)
    assert m.get_option("run_steps") == 0
    assert torch.cuda.mem_get_info(0)[0] == free0
    m.close()


@pytest.mark.parametrize("cells,threads,shares", [(20000, 4, False), (5000, 6, False), (500, 4, True)])
def test_handles_in_several_threads(pkg, cells, threads, shares):
    """Handles stepped from threads: where their tiles do not share the chip, the step's kernels of all of
    them do, and no handle holds it alone; where they do, each takes the run kernel.  The bits are those
    of a handle alone."""
    import threading

    case = pkg.workloads.dam_break(n_cells=cells)
    alone = pkg.SpModel(case)
    alone.prepare()
    alone.step(64)
    assert alone.get_option("run_steps") == 64
    models = [pkg.SpModel(case) for _ in range(threads)]
    for m in models:
        m.prepare()
    start = threading.Barrier(threads)

    def work(m):
        start.wait()
        for _ in range(40):
            m.step(64)

    pool = [threading.Thread(target=work, args=(m,)) for m in models]
    for th in pool:
        th.start()
    for th in pool:
        th.join()
    alone.step(64 * 39)
    share = sum(m.get_option("run_steps") for m in models) / (threads * 40 * 64)
    assert share > 0.9 if shares else share < 0.8      # first and last calls overlap fewer others
    assert all(_same_state(m, alone) and m.time == alone.time for m in models)
    models[0].step(64)                                 # alone again
    assert models[0].get_option("run_steps") >= 64
    for m in models + [alone]:
        m.close()


def test_first_steps_of_a_handle(pkg):
    """A model that takes a few steps does not pay for the run kernel's tiles; one that goes on, is prepared,
    or is told to, has them."""
    case = pkg.workloads.dam_break(n_cells=20000)
    models = [pkg.SpModel(case) for _ in range(4)]
    calls = (1, 30, 40, 10, 5)                     # 78 steps pay for the tiles of 20,000 cells
    taken = []
    models[1].prepare()
    models[2].set_option("run_kernel", 1)
    models[3].set_option("run_kernel", 0)
    for m in models:
        row = []
        for n in calls:
            assert m.step(n) == n
            row.append(m.get_option("run_steps"))
        taken.append(row)
    assert taken == [[0, 0, 0, 10, 15], [1, 31, 71, 81, 86], [1, 31, 71, 81, 86], [0] * 5]
    assert all(_same_state(m, models[0]) and m.time == models[0].time for m in models[1:])
    for m in models:
        m.close()
    m = pkg.SpModel(pkg.workloads.dam_break(n_cells=500))
    m.step(7)                                      # 8 steps pay for the tiles of 500 cells
    assert m.get_option("run_steps") == 0
    m.step(1)
    assert m.get_option("run_steps") == 1
    m.close()


@pytest.mark.parametrize("scheme", ["muscl_evr", "godunov"])
@pytest.mark.parametrize("cells", [800, 20000])
def test_autotuning_times_the_run_kernel(pkg, cells, scheme, tmp_path):
    """The step's autotuner measures the run kernel of a small mesh beside the other forms, keeps it unless
    one of them is faster, and leaves the run's bits alone; with the option 0 it is no candidate."""
    case = pkg.workloads.channel_features(n_cells=cells, scheme=scheme)
    a, b, c = (pkg.SpModel(case) for _ in range(3))
    for m in (a, b, c):
        m.step(25)
    cache = str(tmp_path / "tune.json")
    rep = pkg.tuning.autotune_step(a, iters=2, tile_sizes=(96, 256), cache_path=cache)
    ms = {k: float(v.rstrip("ms")) for k, v in (w.split("=") for w in rep["report"].split() if "=" in w)}
    rest = min(v for k, v in ms.items() if k.startswith(("four-kernel", "fused")))
    kept = ms["run-kernel"] < rest + ms["k_update"]
    assert kept == ("chosen run kernel" in rep["report"]) and (not kept or not rep["fused"])
    before = a.get_option("run_steps")
    assert a.step(50) == b.step(50) == 50
    assert a.get_option("run_steps") - before == (0 if rep["fused"] else 50)
    assert _same_state(a, b) and a.time == b.time
    for name in ("slope_x", "slope_y"):
        if scheme == "muscl_evr" and not rep["fused"]:
            assert np.array_equal(_bits(a.array(name)), _bits(b.array(name)))
    c.set_option("run_kernel", 0)
    assert "run-kernel" not in pkg.tuning.autotune_step(c, iters=2, tile_sizes=(96,), cache_path=cache)["report"]
    for m in (a, b, c):
        m.close()


def test_a_wait_that_ran_out_is_reported_once(pkg):
    """With the state and the time set again the handle goes on, also without a saved point."""
    case = pkg.workloads.dam_break(n_cells=4000)
    a, b = pkg.SpModel(case), pkg.SpModel(case)
    for m in (a, b):
        m.prepare()
    a.set_option("run_wait_polls", 0)
    with pytest.raises(pkg.Sw2dError, match="run kernel ran out"):
        a.step(20)
    a.set_option("run_wait_polls", -1)
    for m in (a, b):
        m.set_state(case.h0 * 1.01, case.q0, case.r0)
        m.set_time(1.0, 0.01)
        assert m.step(20) == 20
    assert _same_state(a, b) and a.time == b.time
    a.close()
    b.close()
