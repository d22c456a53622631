"""A batch whose composition changes between steps: the step that follows launches what a
fresh batch of the same composition launches, and gives its bits."""
import json

import pytest
import torch
from torch.profiler import ProfilerActivity, profile

from nonnewton_b200 import _abi
from nonnewton_b200 import scene as S
from nonnewton_b200.batch import Batch, scene_grid_cells

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


def _kernels(b, path, run=None):
    """Names and grids of the kernels of a step (or of `run`), in time order (none without a profiler)."""
    with profile(activities=[ProfilerActivity.CUDA]) as p:
        run() if run else b.step(1)
        torch.cuda.synchronize()
    p.export_chrome_trace(str(path))
    ev = [e for e in json.loads(path.read_text())["traceEvents"] if e.get("cat") == "kernel"]
    return [(e["name"], e["args"]["grid"]) for e in sorted(ev, key=lambda e: e["ts"])]


# fluid on both sides of every line of the choices: lanes (10,000, 28,000, 56,000 fluid), the list
# build (110,000 slots), the viscosity's one-kernel loop (250,000), its grid (powers of two)
@pytest.mark.parametrize("implicit", [False, True])
def test_choices_follow_the_composition(cuda_lib, tmp_path, implicit):
    """Up and down through the sizes: the launch choices of a captured step (lanes, list build,
    loops in one kernel or as while-nodes, their grids) are those of the present composition,
    not of the one before it or of the one that was captured first."""
    kind = dict(extra_cfg={"useNonNewtonianModel": True},
                fluid_cfg={"nonNewtonMethod": "CROSS_", "viscosity0": 5.0, "viscosity_inf": 0.01,
                           "consistency_index": 1.0, "power_index": 0.7, "viscosityMethod": 13,
                           "viscoMaxError": 1e-5}) if implicit else {}
    scenes = [S.dam_break(seed=k, n_side=(side,) * 3, box=(side + 4) * 0.02, **kind)
              for k, side in enumerate((9, 24, 33, 45, 50, 62))]
    sizes = [sc.particles.n for sc in scenes]
    assert sizes[0] < 2000 and sizes[3] < 110000 < sizes[4] < 250000 < sizes[5]
    cells = max(scene_grid_cells(sc, x_split=2) for sc in scenes)
    b = Batch(sizes[-1], 1, max_cells=cells)
    want = []
    for sc in scenes:
        fresh = Batch(sizes[-1], 1, max_cells=cells)
        fresh.set([sc])
        want.append((_steps(fresh), _kernels(fresh, tmp_path / "trace.json")))
        fresh.engine.close()
    for k in (0, 1, 2, 3, 4, 5, 4, 5, 3, 2, 0, 4, 1):
        b.set([scenes[k]])
        _same(_steps(b), want[k][0])
        assert _kernels(b, tmp_path / "trace.json") == want[k][1]


def test_launch_counts_across_compositions(cuda_lib, tmp_path):
    """nn_launch_count over steps of several compositions and a pass of its own: the kernels that
    a profiler sees (small scenes, whose loops are no while-nodes)."""
    kind = dict(extra_cfg={"useNonNewtonianModel": True},
                fluid_cfg={"nonNewtonMethod": "CROSS_", "viscosity0": 5.0, "viscosity_inf": 0.01, "consistency_index": 1.0,
                           "power_index": 0.7, "viscosityMethod": 13})
    scenes = [S.dam_break(seed=1, n_side=(8, 7, 6), box=0.4), S.dam_break(seed=2, n_side=(9, 8, 7), box=0.4, **kind)]
    b = Batch(8000, 1)
    first = b.engine.launch_count()
    seen = in_set = 0
    for k in (0, 1, 0, 1):
        before = b.engine.launch_count()
        b.set([scenes[k]])
        in_set += b.engine.launch_count() - before
        seen += len(_kernels(b, tmp_path / "trace.json"))
        seen += len(_kernels(b, tmp_path / "trace.json"))
    seen += len(_kernels(b, tmp_path / "trace.json", lambda: b.engine.run_pass(_abi.NN_PASS_SUBSTEP)))
    if seen:  # a profiler is there
        assert b.engine.launch_count() - first == in_set + seen
