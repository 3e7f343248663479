"""A gradient after a change of the parameters runs the trajectory itself and keeps the steps of its
last segments; after replay_cost the checkpoints are valid and every segment is recomputed.  The two
give the same bits, whatever number of segments is kept."""
import numpy as np
import pytest

from tests.conftest import load_pkg

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def pkg():
    return load_pkg()


def _bits(out):
    J, g = out
    return [np.float64(J).view(np.int64)] + [np.asarray(g[k]).view(np.int64) for k in sorted(g)]


# steps and interval: several segments, a short last one, one step per segment, one segment only, and a
# trajectory that t_max cuts short (of the 60 steps asked for)
@pytest.mark.parametrize("steps,every,t_max", [(60, 16, None), (45, 15, None), (7, 1, None), (20, 64, None), (60, 16, 0.4)])
@pytest.mark.parametrize("scheme", ["muscl_evr", "godunov"])
def test_kept_steps_give_the_same_gradient(pkg, scheme, steps, every, t_max):
    case = pkg.workloads.dam_break(n_cells=2500, scheme=scheme)
    rng = np.random.default_rng(7)
    friction = case.friction[0] * (1.0 + 0.1 * rng.uniform(-1, 1, case.h0.size))
    if t_max is not None:
        probe = pkg.SpModel(case)
        probe.step(steps)
        case.opts = dict(case.opts, t_max=t_max * probe.time[0])
    want = None
    for kept in (None, 1, 2, 3):
        model = pkg.SpModel(case)
        if kept:
            model.set_option("adjoint_kept_segments", kept)
        n = model.record(steps, every)
        assert (n < steps) == (t_max is not None)
        cells = np.sort(rng.choice(model.n, size=16, replace=False)) if want is None else cells
        at = np.unique(np.linspace(0, n, 5).astype(int))
        model.set_observations(cells, at, np.tile(case.h0[cells] * 1.02, (at.size, 1)))
        model.set_param("friction", friction)
        first = _bits(model.adjoint())     # runs the trajectory
        again = _bits(model.adjoint())     # its checkpoints are valid: recomputes
        model.set_param("friction", friction)
        J = model.replay_cost()
        after = _bits(model.adjoint())
        want = want or after
        for out in (first, again, after):
            assert all(np.array_equal(a, b) for a, b in zip(out, want))
        assert np.float64(J).view(np.int64) == want[0]


def test_kept_segments_option(pkg):
    model = pkg.SpModel(pkg.workloads.dam_break(n_cells=400))
    with pytest.raises(pkg.Sw2dError):
        model.set_option("adjoint_kept_segments", 0)


def test_recording_again_and_closing(pkg):
    """The kept buffers go with the trajectory: handles that record again, or are closed, leave the
    others' gradients alone."""
    case = pkg.workloads.dam_break(n_cells=1500)

    def observe(model, n):
        model.set_observations([3, 40], [n // 2, n], np.full((2, 2), 1.0))
        model.set_param("friction", case.friction[0] * 1.1)
        return _bits(model.adjoint())

    a, b = pkg.SpModel(case), pkg.SpModel(case)
    for model in (a, b):
        model.record(30, 8)
    want = observe(a, 30)
    assert all(np.array_equal(x, y) for x, y in zip(observe(b, 30), want))
    c = pkg.SpModel(case)
    c.record(12, 3)
    c.close()
    a.close()
    assert all(np.array_equal(x, y) for x, y in zip(observe(b, 30), want))
