"""A batch whose composition changes between steps: the step that follows launches what a
fresh batch of the same composition launches, and gives its bits."""
import pytest
import torch

from nonnewton_b200 import scene as S
from nonnewton_b200.batch import Batch

pytestmark = pytest.mark.gpu
FIELDS = ("x", "v", "acceleration", "density", "volume")


def _steps(b, n=2):
    """Steps from the packed state; the kernel launches of the last of them and the fields."""
    b.step(n)
    before = b.engine.launch_count()
    b.step(1)
    launches = b.engine.launch_count() - before
    assert all(b.stats(k)["status"] == 0 for k in range(len(b.scenes)))
    return launches, [b.scene_view(k, f).clone() for k in range(len(b.scenes)) for f in FIELDS]


def _same(a, b):
    assert a[0] == b[0]
    for x, y in zip(a[1], b[1]):
        assert torch.equal(x, y)


def _rigid(seed, bodies=1):
    sc = S.rigid_drop(seed=seed, n_body=(4, 3, 4))
    if bodies == 2:  # the upper half of the body as a body of its own
        rb = sc.particles.phase_id == 2000
        y = sc.particles.x[:, 1]
        sc.particles.phase_id[rb & (y > y[rb].mean())] = 2001
    return sc


@pytest.mark.parametrize("capacity", [8000, 9000])  # the bodies' one-block kernel, the separate ones
@pytest.mark.parametrize("bodies,then", [(1, 0), (2, 1), (2, 0)])
def test_rigid_bodies_leave_the_batch(cuda_lib, capacity, bodies, then):
    """The launches of the bodies and the addresses of their tables are part of a captured
    step: a set without bodies, or with fewer, takes none of them from the set before it."""
    after = _rigid(4, then) if then else S.dam_break(seed=3, n_side=(9, 8, 7), box=0.4)
    b = Batch(capacity, 2)
    b.set([_rigid(2, bodies)])
    _steps(b)
    b.set([after])
    fresh = Batch(capacity, 2)
    fresh.set([after])
    got, want = _steps(b), _steps(fresh)
    if then:  # the bodies' sums are FP64 atomics: positions agree to an ulp or two at the domain's size
        assert got[0] == want[0] and (got[1][0] - want[1][0]).abs().max() <= 2e-7
    else:
        _same(got, want)


def test_rigid_scene_is_repacked_away(cuda_lib):
    dam = S.dam_break(seed=3, n_side=(9, 8, 7), box=0.4)
    b = Batch(8000, 2)
    b.set([_rigid(2), dam])
    _steps(b)
    b.repack([1], [])
    fresh = Batch(8000, 2)
    fresh.set([dam])
    _steps(fresh)
    fresh.repack([0], [])
    _same(_steps(b), _steps(fresh))
