"""Engine.neighbors for fewer rows than there are particles, and for more."""
import pytest
import torch

from nonnewton_b200 import scene as S
from nonnewton_b200 import sph
from nonnewton_b200.config import SimConfig

pytestmark = pytest.mark.gpu


def test_fewer_and_more_rows_than_particles(cuda_lib):
    sc = S.dam_break(seed=1, n_side=(7, 6, 5), box=0.3)
    m = sph.initialize(SimConfig(config=sc.config), particles=sc.particles)
    m.ns.run_search()
    n = sc.particles.n
    num, lists = m.engine.neighbors(n, 40)
    for k in (0, 1, 33, n, n + 5):
        a, b = m.engine.neighbors(k, 40)
        assert a.shape == (k,) and b.shape == (k, 40) and b.is_contiguous()
        assert torch.equal(a[:n], num[:k]) and torch.equal(b[:n], lists[:k])
        assert not bool(a[n:].any()) and bool((b[n:] == -1).all())
