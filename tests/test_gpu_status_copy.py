"""nn_status_async into mapped pinned memory (written by a kernel) and into pageable memory
(copied): the values that the scene's statistics report, also behind a step still running."""
import pytest
import torch

from nonnewton_b200 import scene as S
from nonnewton_b200 import sph
from nonnewton_b200.config import SimConfig

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pinned", [True, False])
@pytest.mark.parametrize("cap", [64, 8])  # 8 overflows
def test_status_copy(cuda_lib, pinned, cap):
    sc = S.dam_break(seed=1, n_side=(9, 8, 7), box=0.4)
    m = sph.initialize(SimConfig(config=sc.config), particles=sc.particles, max_neighbors=cap)
    solver = sph.build_solver()
    solver.grow_neighbors = False
    out = torch.full((6,), -7, dtype=torch.int32, pin_memory=pinned)
    m.engine.step(2)
    m.engine.status_async(out[2:4])  # an offset into the allocation
    m.engine.status_wait()
    st = m.engine.stats(0)
    assert out.tolist() == [-7, -7, st["status"], st["max_neighbors_seen"], -7, -7]
    assert (st["status"] != 0) == (cap == 8) and st["max_neighbors_seen"] > 8
