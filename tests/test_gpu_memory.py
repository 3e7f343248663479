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

    # slopes (MUSCL-EVR), Riemann states, the edges' sides, and the kept segments
    assert _failing_in_turn(pkg, lambda: pkg.SpModel(case), act) >= (3 + 1 if scheme == "muscl_evr" else 2 + 1)


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


def _recorded(pkg, case):
    model = pkg.SpModel(case)
    model.record(20, 6)
    model.set_observations([3, 50], [10, 20], np.full((2, 2), 1.0))
    return model


def _gradient(model, friction):
    model.set_param("friction", friction)
    J, g = model.adjoint()
    return [np.float64(J)] + [g[k] for k in sorted(g)]


def _assimilating(pkg, case, dt):
    model = pkg.SpModel(case)
    model.assim_configure(phi_transform="none", cost_normalize=True)
    model.assim_set_gauges([8 * dt, 16 * dt], [3, 50], np.ones(2), np.full((2, 2), 1.0))
    return model


def test_kept_memory_gives_way(pkg):
    """The kept steps of one handle and the kept slopes of another go to whatever finds no room: a
    model's creation, a record, a network's training buffers.  The next gradients take them again, with
    the same results; those of a handle that cannot, too."""
    case = pkg.workloads.dam_break(n_cells=600)
    free = pkg.workloads.dam_break(n_cells=600, friction="none")
    probe = pkg.SpModel(free)
    probe.step(3)
    dt = probe.dt
    probe.close()
    free.opts = dict(free.opts, t_max=20 * dt)
    fails = pkg.capi.load_library().sw2d_test_fail_allocations
    a, b = _recorded(pkg, case), _assimilating(pkg, free, dt)
    want_a, want_b = _gradient(a, case.friction[0] * 1.1), b.assim_gradient(free.phi, 6)[0]
    held = a.get_option("kept_bytes"), b.get_option("kept_bytes")
    assert held[0] > 0 and held[1] > 0
    net = pkg.closure.MLP(pkg.closure.init_params(0))
    x, t = np.zeros((300, 10), np.float32), np.zeros((300, 2), np.float32)

    for other in (lambda: pkg.SpModel(case).close(), lambda: _recorded(pkg, case).close(), lambda: net.loss_grad(x, t)):
        fails(0, 1)
        try:
            other()
        finally:
            fails(0, 0)
        assert (a.get_option("kept_bytes"), b.get_option("kept_bytes")) == (0, 0)
        got = _gradient(a, case.friction[0] * 1.1)
        assert all(np.array_equal(_bits(x), _bits(y)) for x, y in zip(got, want_a))
        assert np.array_equal(_bits(b.assim_gradient(free.phi, 6)[0]), _bits(want_b))
        assert (a.get_option("kept_bytes"), b.get_option("kept_bytes")) == held
    # taken back and not to be had again: every segment recomputed, the slopes rebuilt
    fails(0, 1)
    pkg.SpModel(case).close()
    for model, act, want in ((a, lambda: _gradient(a, case.friction[0] * 1.1), want_a),
                             (b, lambda: [b.assim_gradient(free.phi, 6)[0]], [want_b])):
        n = fails(0, 0)
        act()
        n = fails(0, 0)                  # the gradient's requests, the kept memory's among them
        fails(0, 1)
        pkg.SpModel(case).close()
        fails(0, n)
        try:
            got = act()
        finally:
            fails(0, 0)
        assert model.get_option("kept_bytes") == 0
        act()                            # and later it is
        assert model.get_option("kept_bytes") == held[model is b]
        assert all(np.array_equal(_bits(x), _bits(y)) for x, y in zip(got, want))
    net.close()
    a.close()
    b.close()


def test_kept_memory_of_several_threads(pkg):
    """Gradients of several handles in threads, while others' allocations take what is idle."""
    import threading

    case = pkg.workloads.dam_break(n_cells=600)
    fails = pkg.capi.load_library().sw2d_test_fail_allocations
    models = [_recorded(pkg, case) for _ in range(4)]
    want = _gradient(models[0], case.friction[0] * 1.1)
    bad = []

    def gradients(m):
        for _ in range(30):
            got = _gradient(m, case.friction[0] * 1.1)
            if not all(np.array_equal(_bits(x), _bits(y)) for x, y in zip(got, want)):
                bad.append(m)

    def creations():
        for _ in range(30):
            fails(0, 1)
            try:
                pkg.SpModel(case).close()
            except pkg.Sw2dError:
                pass                     # nothing was idle
            finally:
                fails(0, 0)

    threads = [threading.Thread(target=gradients, args=(m,)) for m in models] + [threading.Thread(target=creations)]
    for th in threads:
        th.start()
    for th in threads:
        th.join()
    assert not bad
    for m in models:
        m.close()


def test_training_buffers(pkg):
    """A batch too large for the memory there is: reported, and batches of the sizes before train on, with
    the gradient of the last one for the next step.  Growing batches keep one set of buffers."""
    import torch

    C = pkg.closure
    fails = pkg.capi.load_library().sw2d_test_fail_allocations
    rng = np.random.default_rng(1)
    x, t = rng.normal(size=(60000, 10)).astype(np.float32), rng.normal(size=(60000, 2)).astype(np.float32)

    def step(net, n):
        loss, g = net.loss_grad(x[:n], t[:n])
        net.adam_step(1e-3)
        return [np.float64(loss), np.asarray(g, np.float64), np.asarray(net.params, np.float64)]

    net, ref = C.MLP(C.init_params(3)), C.MLP(C.init_params(3))
    assert all(np.array_equal(a, b) for a, b in zip(step(net, 300), step(ref, 300)))
    fails(0, 0)
    C.MLP(C.init_params(3)).loss_grad(x[:1], t[:1])
    n = fails(0, 0)
    tried = 0
    for skip in range(n):
        fails(skip, 1)
        try:
            net.loss_grad(x[:5000], t[:5000])
            break                        # fewer requests than a first batch makes
        except RuntimeError:
            tried += 1
        finally:
            fails(0, 0)
        net.adam_step(1e-3)              # the gradient of the last batch is still there
        ref.adam_step(1e-3)
        assert np.array_equal(net.params, ref.params)
        assert all(np.array_equal(a, b) for a, b in zip(step(net, 300), step(ref, 300)))
    assert tried >= 5
    free = []
    for k in range(6):
        net.loss_grad(x[:50000 + 1000 * k], t[:50000 + 1000 * k])
        free.append(torch.cuda.mem_get_info(0)[0])
    assert free[0] - free[-1] <= 4 << 20       # the last set is 10 % larger than the first, no more
    net.close()
    ref.close()


def test_kept_segments_are_one_allocation(pkg):
    case = pkg.workloads.dam_break(n_cells=600)
    fails = pkg.capi.load_library().sw2d_test_fail_allocations
    requests = []
    for kept in (1, 3):
        model = pkg.SpModel(case)
        model.set_option("adjoint_kept_segments", kept)
        fails(0, 0)
        model.record(20, 6)
        requests.append(fails(0, 0))
        model.close()
    assert requests[1] == requests[0] + 1


def test_training_without_pinned_memory(pkg):
    """A first batch requests five device buffers, then pinned memory for its result, which ordinary memory
    replaces where there is none; a larger batch asks again."""
    C = pkg.closure
    fails = pkg.capi.load_library().sw2d_test_fail_allocations
    rng = np.random.default_rng(2)
    x, t = rng.normal(size=(900, 10)).astype(np.float32), rng.normal(size=(900, 2)).astype(np.float32)
    a, b = C.MLP(C.init_params(3)), C.MLP(C.init_params(3))
    for n in (300, 200, 900):
        out = []
        for net, first in ((a, 5), (b, 0)):
            fails(first, 1 if net is a and n == 300 else 0)
            loss, g = net.loss_grad(x[:n], t[:n])
            assert fails(0, 0) == {300: 6, 200: 0}.get(n, 6)
            net.adam_step(1e-3)
            out.append((loss, g, net.params))
        assert out[0][0] == out[1][0] and all(np.array_equal(u, v) for u, v in zip(out[0][1:], out[1][1:]))
    a.close()
    b.close()
