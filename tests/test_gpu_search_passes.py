"""The search's scan (16,384 counts a tile, 16-byte loads, a ragged end) and its in-cell sort
(registers up to 16 particles, in place up to 24, a warp above): lists against brute force
over grids on both sides of a tile, and slot orders that do not depend on the atomics."""
import numpy as np
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


def test_slot_order_of_crowded_cells(cuda_lib):
    """Cells of 1 to 34 particles: three steps (the first sorts the caller's order, the others
    the previous slots) give the same bits every time, so the order in a cell is the ids'."""
    sc = S.dam_break(seed=2, n_side=(14, 11, 9), box=0.5)
    x, nf, rng = sc.particles.x, sc.particles.n_fluid, np.random.default_rng(4)
    ids, at = rng.permutation(nf), 0
    for k in range(1, 35):
        c = np.array([3 + k % 7, 2 + k // 7, 8], np.float32) * 0.04  # a cell's lower corner
        x[ids[at:at + k]] = c + rng.uniform(0.005, 0.035, (k, 3)).astype(np.float32)
        at += k
    out = []
    for _ in range(4):
        m = sph.initialize(SimConfig(config=sc.config), particles=sc.particles, max_neighbors=256)
        solver = sph.build_solver()
        solver.initialize()
        m.engine.step(3)
        out.append([m.pd.x.clone(), m.pd.v.clone(), m.pd.density.clone()])
    for o in out[1:]:
        for a, b in zip(o, out[0]):
            assert torch.equal(a, b)
