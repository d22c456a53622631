"""In a cell, slots follow the particle ids, also where a step starts from the previous slots and
the cell's particles come from two cells: sums over neighbours, which follow the slots, have the
bits of a step that starts from the caller's arrays (there the source index is the id)."""
import numpy as np
import pytest
import torch

from nonnewton_b200 import scene as S
from nonnewton_b200 import sph
from nonnewton_b200.config import SimConfig

pytestmark = pytest.mark.gpu


def _clusters():
    """Clusters of 1 to 34 dynamic solid particles, one per cell and apart from each other, half
    of each a cell further along x, from where a step takes it in. Ids are shuffled."""
    sc = S.dam_break(seed=1, n_side=(2, 2, 2), box=1.2)
    p = sc.param
    edge = p.support_radius * (1 + 1e-3)
    rng = np.random.default_rng(3)
    x, move, cell = [], [], []
    for k in range(1, 35):
        corner = np.array([4 + 4 * (k % 6), 5 + 4 * ((k // 6) % 6), 7]) * edge + (p.domain_start - 2 * p.support_radius)
        x.append(corner + rng.uniform(0.1, 0.9, (k, 3)) * edge)
        move.append(np.arange(k) % 2 == 1)
        cell.append(np.full(k, k))
    ids = rng.permutation(sum(range(1, 35)))
    x, move, cell = np.concatenate(x)[ids], np.concatenate(move)[ids], np.concatenate(cell)[ids]
    n = len(x)
    start = x + np.array([edge, 0, 0]) * move[:, None]
    v = np.array([-edge / p.dt, 0, 0]) * move[:, None]
    ps = S.ParticleSet(x=start.astype(np.float32), material=np.full(n, S.SOLID, np.int32),
                       is_dynamic=np.ones(n, np.int32), phase_id=np.full(n, 1000, np.int32),
                       mass=np.full(n, p.volume0 * p.density0, np.float32), n_fluid=0)
    sc.config["Configuration"]["gravitation"] = [0.0, 0.0, 0.0]
    return sc, ps, v.astype(np.float32), cell, edge


def test_slots_of_a_cell_follow_the_ids(cuda_lib):
    sc, ps, v, cluster, edge = _clusters()
    out = []
    for resume in (False, True):
        m = sph.initialize(SimConfig(config=sc.config), particles=ps, max_neighbors=64, tuning=dict(x_split=1))
        solver = sph.build_solver()
        solver.initialize()
        m.pd.v.copy_(torch.from_numpy(v))
        m.engine.step(1)
        x = m.pd.x.cpu().numpy()
        m.engine.step(1, resume=resume)
        assert solver.stats()["status"] == 0
        out.append([getattr(m.pd, f).clone() for f in ("volume", "x", "v")])
    # the second search met every cluster whole, in a cell of its own
    at = np.floor((x - (sc.param.domain_start - 2 * sc.param.support_radius)) / edge).astype(int)
    for k in range(1, 35):
        assert len(np.unique(at[cluster == k], axis=0)) == 1
    assert len(np.unique(at, axis=0)) == 34
    for a, b in zip(*out):
        assert torch.equal(a, b)
