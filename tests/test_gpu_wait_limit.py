"""A wait inside a one-kernel solver loop that runs out: the kernel returns, every scene of the
batch reports it, the object API raises, and the step after it starts with a barrier at rest.
The limit of 0 polls makes each block that is not the last to arrive give up at once."""
import pytest
import torch

from nonnewton_b200 import _abi
from nonnewton_b200 import scene as S
from nonnewton_b200 import sph
from nonnewton_b200.batch import Batch
from nonnewton_b200.config import SimConfig
from nonnewton_b200.engine import NNError

pytestmark = pytest.mark.gpu
CROSS = dict(extra_cfg={"useNonNewtonianModel": True},
             fluid_cfg={"nonNewtonMethod": "CROSS_", "viscosity0": 5.0, "viscosity_inf": 0.01, "consistency_index": 1.0,
                        "power_index": 0.7, "viscosityMethod": 13, "viscoMaxError": 1e-5})


def _bodies(b, k):
    st = b.stats(k)
    return st["iterations_v"], st["iterations"], st["cg_iterations"]


@pytest.mark.parametrize("kind,side", [({}, 9), (CROSS, 11), (CROSS, 16)])  # 8 lanes, 4 with three scenes
def test_every_scene_reports_it_and_the_next_step_recovers(cuda_lib, kind, side):
    scenes = [S.dam_break(seed=k, n_side=(side, side + k, side), box=(side + 5) * 0.02, **kind) for k in range(3)]
    n = sum(sc.particles.n for sc in scenes)
    b, fresh = Batch(n, 3), Batch(n, 3)
    b.set(scenes)
    fresh.set(scenes)
    b.engine.set_wait_limit(0)
    b.step(1)
    assert [b.stats(k)["status"] for k in range(3)] == [_abi.NN_ERR_CUDA] * 3
    b.engine.set_wait_limit(None)
    b.set(scenes)
    b.step(3)
    fresh.step(3)
    for k in range(3):
        assert b.stats(k)["status"] == 0 and _bodies(b, k) == _bodies(fresh, k)
        for f in ("x", "v", "density"):
            assert torch.equal(b.scene_view(k, f), fresh.scene_view(k, f))
    # without setting the scenes again: the barrier is at rest, the status stays
    b.engine.set_wait_limit(0)
    b.step(1)
    b.engine.set_wait_limit(None)
    for f in ("x", "x_0", "v", "acceleration", "density", "volume", "dfsph_factor", "density_adv"):
        getattr(b.pd, f).copy_(getattr(fresh.pd, f))
    b.step(2)
    fresh.step(2)
    for k in range(3):
        assert b.stats(k)["status"] == _abi.NN_ERR_CUDA and _bodies(b, k) == _bodies(fresh, k)
        # (which body carried the force terms, and so their rounding, follows the step before)
        for f, tol in (("x", 2e-7), ("v", 1e-5)):
            assert (b.scene_view(k, f) - fresh.scene_view(k, f)).abs().max() <= tol


def test_the_solver_raises(cuda_lib):
    sc = S.dam_break(seed=1, n_side=(9, 8, 7), box=0.4)
    for checked_at_once in (True, False):
        m = sph.initialize(SimConfig(config=sc.config), particles=sc.particles, max_neighbors=64 if checked_at_once else 200)
        solver = sph.build_solver()
        solver.initialize()
        if not checked_at_once:  # the copy of the status is checked by the next call
            solver.step()
            solver.step()
            assert solver._pending is not None
        m.engine.set_wait_limit(0)
        if checked_at_once:
            with pytest.raises(NNError) as e:
                solver.step()
        else:
            solver.step()
            with pytest.raises(NNError) as e:
                solver.step()
        assert e.value.code == _abi.NN_ERR_CUDA
        assert solver.stats()["status"] == _abi.NN_ERR_CUDA
