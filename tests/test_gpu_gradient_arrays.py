"""sw2d_get_array("slope_x" / "slope_y") after a gradient.  sw2d_adjoint leaves the model at the
trajectory's end, so the arrays of the last step are those of the trajectory's last step at the
current parameters, which sw2d_replay_cost (it runs the same steps and keeps none) leaves too."""
import numpy as np
import pytest

from tests.conftest import load_pkg

pytestmark = pytest.mark.gpu


# segments: several, one, the last one short; kept: all of them, the last one only
@pytest.mark.parametrize("steps,every", [(40, 10), (12, 64), (23, 5)])
@pytest.mark.parametrize("kept", [None, 1])
def test_slopes_of_the_last_step(steps, every, kept):
    pkg = load_pkg()
    case = pkg.workloads.dam_break(n_cells=2500)
    model = pkg.SpModel(case)
    if kept:
        model.set_option("adjoint_kept_segments", kept)
    n = model.record(steps, every)
    cells = np.arange(5, model.n, 97)
    model.set_observations(cells, [n // 2, n], np.tile(case.h0[cells] * 1.05, (2, 1)))
    recorded = model.array("slope_x")
    model.set_param("friction", case.friction[0] * 2.0)
    model.replay_cost()
    want = [model.array(name) for name in ("slope_x", "slope_y")]
    model.set_param("friction", case.friction[0])    # another trajectory in between
    model.replay_cost()
    assert not np.array_equal(want[0], recorded) and np.array_equal(model.array("slope_x"), recorded)
    model.set_param("friction", case.friction[0] * 2.0)
    model.adjoint()
    for name, w in zip(("slope_x", "slope_y"), want):
        assert np.array_equal(model.array(name), w), name
    model.close()
