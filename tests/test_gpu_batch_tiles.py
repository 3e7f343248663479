"""The work queue's default tile (queue_tile_rule): the measured best, or within 1 % of it, at ensembles
from 22k cells to 2.5M on a GPU of 148 SMs."""
import pytest

from tests.conftest import load_pkg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("members,cells,tile", [(6, 3700, 128), (24, 25000, 512), (8, 150000, 1024), (12, 143000, 1024),
                                                (16, 156000, 2048)])
def test_default_tile(members, cells, tile):
    import torch

    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("measured on 148 SMs")
    pkg = load_pkg()
    case = pkg.workloads.dam_break(n_cells=cells)
    models = [pkg.SpModel(case) for _ in range(members)]
    batch = pkg.Batch(models)
    assert batch.config["cells_per_tile"] == batch.config["edges_per_tile"] == tile
    assert list(batch.step(2)) == [2] * members
    batch.close()
    for m in models:
        m.close()
