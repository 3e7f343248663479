"""Loss and gradient of the closure network at batch sizes around the training kernel's tile (128
rows) and its persistent grid (one CTA per SM), against the FP64 reference with the same BF16
roundings.  The kernel differs from it by FP32 accumulation (far below) and by the hardware tanh,
which moves an activation or a back-propagated value by at most one BF16 unit (2^-8 relative)."""
import numpy as np
import pytest

from tests.conftest import load_pkg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 127, 128, 129, 1000, 148 * 128, 148 * 128 + 1, 40003])
def test_loss_and_gradient_at_tile_edges(n):
    p = load_pkg()
    p.build.build()
    C = p.closure
    rng = np.random.default_rng(n)
    norm = np.concatenate([rng.normal(0, 1, 10), rng.uniform(0.5, 2, 10), rng.normal(0, 1, 2),
                           rng.uniform(0.5, 2, 2)]).astype(np.float32)
    x = (rng.normal(0, 1.5, (n, 10)) * norm[10:20] + norm[:10]).astype(np.float32)
    t = rng.normal(0, 1, (n, 2)).astype(np.float32) * norm[22:24] + norm[20:22]
    params = C.init_params(n % 7)
    params[640:704] = rng.normal(0, 0.2, 64)
    net = C.MLP(params, norm)
    loss, g = net.loss_grad(x, t)
    rloss, rg = C.reference_loss_grad(params, norm, x, t)
    unit = 2.0 ** -8
    assert abs(loss - rloss) <= unit * rloss
    k = 0
    for name, shape in C.SHAPES:
        m = int(np.prod(shape))
        assert np.linalg.norm(g[k:k + m] - rg[k:k + m]) <= unit * np.linalg.norm(rg[k:k + m]), name
        k += m
    again, g2 = net.loss_grad(x, t)          # the same batch again: the same bits
    assert again == loss and np.array_equal(g.view(np.int32), g2.view(np.int32))
    net.close()


def test_training_wait_that_runs_out():
    """A first wait that gives up at once: the training kernel drains the MMA in flight, frees its
    TMEM and reports; the network then trains as before."""
    C = load_pkg().closure
    rng = np.random.default_rng(1)
    x, t = rng.normal(size=(300, 10)).astype(np.float32), rng.normal(size=(300, 2)).astype(np.float32)
    net = C.MLP(C.init_params(3))
    loss, g = net.loss_grad(x, t)
    net.set_wait_polls(0)
    with pytest.raises(RuntimeError, match="tensor-core wait ran out"):
        net.loss_grad(x, t)
    net.set_wait_polls(-1)
    again, g2 = net.loss_grad(x, t)
    assert again == loss and np.array_equal(g.view(np.int32), g2.view(np.int32))
    net.close()
