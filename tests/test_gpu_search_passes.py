"""The search's scan (16,384 counts a tile, 16-byte loads, a ragged end): lists against brute
force over grids on both sides of a tile."""
import pytest
import torch

from nonnewton_b200 import scene as S
from nonnewton_b200 import sph
from nonnewton_b200.config import SimConfig

pytestmark = pytest.mark.gpu


# gx * 4^m cells: 13..18 x 1,024 (one tile is 16 x 1,024), 25 x 1,024, 33+ x 4,096
@pytest.mark.parametrize("box", [0.42, 0.5, 0.53, 0.56, 0.6, 0.9, 1.25])
def test_lists_over_grid_sizes(cuda_lib, box):
    sc = S.dam_break(seed=1, n_side=(6, 7, 5), box=box)
    m = sph.initialize(SimConfig(config=sc.config), particles=sc.particles)
    m.ns.run_search()
    num, lists = m.engine.neighbors(len(sc.particles.x), 64)
    xt = m.pd.x
    r2 = torch.zeros(len(xt), len(xt), device="cuda")
    for k in range(3):
        e = xt[:, None, k] - xt[None, :, k]
        r2 = r2 + e * e
    near = r2.sqrt() < torch.tensor(sc.param.support_radius, dtype=torch.float32, device="cuda")
    near.fill_diagonal_(False)
    want = torch.full((len(xt), 64), -1, dtype=torch.int32, device="cuda")
    i, j = near.nonzero(as_tuple=True)
    want[i, torch.arange(len(i), device="cuda") - (near.sum(1).cumsum(0) - near.sum(1))[i]] = j.int()
    assert torch.equal(num, near.sum(1).int()) and torch.equal(lists, want)
