"""The launch variants of the DDP edge kernel, which the mesh size chooses among, give the same bits."""
import numpy as np
import pytest

from tests.conftest import load_pkg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("laws", ["linear", "mixed"])
def test_ddp_edge_variants_agree(laws):
    pkg = load_pkg()
    want = None
    for variant in range(6):
        model = pkg.SpModel(pkg.workloads.ddp_channel(n_cells=3000, laws=laws, moving=True))
        model._check(model.lib.sw2d_set_launch_config(model.handle, 4, variant))
        model.step(40)
        got = [np.asarray(a).view(np.int64) for a in model.state()]
        want = want or got
        assert all(np.array_equal(a, b) for a, b in zip(got, want)), variant
