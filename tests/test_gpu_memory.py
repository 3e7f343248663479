"""Device memory that only saves time (the kept steps and slopes of the gradients) and memory that a
call needs, when the device has none left: allocations failing one by one
(sw2d_test_fail_allocations), in turn."""
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


def _failing_in_turn(pkg, make, act):
    """act(make()) with each of its allocations failing in turn: how many of them it did without, each
    time with the same result."""
    fails = pkg.capi.load_library().sw2d_test_fail_allocations
    model = make()
    fails(0, 0)
    want = act(model)
    n = fails(0, 0)
    model.close()
    served = 0
    for skip in range(n):
        model = make()
        fails(skip, 1)
        try:
            got = act(model)
        except pkg.Sw2dError:
            got = None               # one that it needs
        finally:
            fails(0, 0)
        if got is not None:
            served += 1
            assert len(got) == len(want) and all(np.array_equal(_bits(a), _bits(b)) for a, b in zip(got, want)), skip
        model.close()
    return served


@pytest.mark.parametrize("scheme", ["muscl_evr", "godunov"])
def test_gradient(pkg, scheme):
    case = pkg.workloads.dam_break(n_cells=600, scheme=scheme)

    def act(model):
        model.record(20, 6)
        model.set_observations([3, 50], [10, 20], np.full((2, 2), 1.0))
        model.set_param("friction", case.friction[0] * 1.1)
        J, g = model.adjoint()
        return [np.float64(J)] + [g[k] for k in sorted(g)]

    # slopes (MUSCL-EVR), Riemann states, the edges' sides, and the kept segments' arrays
    assert _failing_in_turn(pkg, lambda: pkg.SpModel(case), act) >= (3 + 4 if scheme == "muscl_evr" else 2 + 3)


@pytest.mark.parametrize("scheme", ["muscl_evr", "godunov"])
def test_porosity_gradient(pkg, scheme):
    case = pkg.workloads.dam_break(n_cells=600, scheme=scheme, friction="none")
    probe = pkg.SpModel(case)
    probe.step(3)
    dt = probe.dt
    probe.close()
    case.opts = dict(case.opts, t_max=20 * dt)

    def make():
        model = pkg.SpModel(case)
        model.assim_configure(phi_transform="none", cost_normalize=True)
        model.assim_set_gauges([8 * dt, 16 * dt], [3, 50], np.ones(2), np.full((2, 2), 1.0))
        return model

    def act(model):
        model.assim_record(case.phi, 6)
        return [model.assim_gradient(case.phi, 6)[0], np.float64(model.assim_replay_cost(case.phi))]

    assert _failing_in_turn(pkg, make, act) >= (1 if scheme == "muscl_evr" else 0)
