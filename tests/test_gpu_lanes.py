"""The lane split of the neighbour passes (nb_sum): contexts pick 8, 4, 2 or 1 lanes per
particle by their fluid count, and every split folds a particle's terms in list order, so
the fields are the one-lane passes' (an explicit unroll) bit for bit: odd sizes on both
sides of each line of the rule, and every pass (explicit and implicit viscosity, the
folded non-pressure terms, a rigid body's coupling)."""
import numpy as np
import pytest
import torch

from nonnewton_b200 import scene as S
from nonnewton_b200 import sph
from nonnewton_b200.config import SimConfig

pytestmark = pytest.mark.gpu
FIELDS = ("x", "v", "acceleration", "density", "volume")
CROSS = dict(extra_cfg={"useNonNewtonianModel": True},
             fluid_cfg={"nonNewtonMethod": "CROSS_", "viscosity0": 5.0, "viscosity_inf": 0.01, "consistency_index": 1.0,
                        "power_index": 0.7, "viscosityMethod": 13, "viscoMaxError": 1e-3, "viscosityBoundary": 0.1})


def _run(sc, unroll):
    m = sph.initialize(SimConfig(config=sc.config), particles=sc.particles, quirks=sc.param.quirks,
                       tuning=dict(unroll=unroll))
    solver = sph.build_solver()
    solver.initialize()
    g = torch.Generator("cuda").manual_seed(1)
    v = torch.rand(m.pd.v.shape, generator=g, device="cuda") - 0.5
    m.pd.v.copy_(v * m.pd.is_dynamic[:, None])
    for _ in range(3):
        solver.step()
    assert solver.stats()["status"] == 0
    nf = sc.particles.n_fluid
    law = ("strain_rate_norm", "nonnewton_viscosity") if sc.param.use_nonnewtonian else ()  # else not written
    out = {k: getattr(m.pd, k).clone() for k in FIELDS + law}
    out.update({k: getattr(m.pd, k)[:nf].clone() for k in ("dfsph_factor", "density_adv")})
    return out


@pytest.mark.parametrize("counts,kind", [((1, 1, 1), {}), ((5, 3, 1), CROSS), ((11, 13, 9), CROSS), ((25, 20, 20), {}),
                                         ((25, 21, 19), CROSS), ((29, 31, 31), {}), ((39, 37, 31), CROSS),
                                         ((39, 39, 37), {})])
def test_sums_do_not_depend_on_the_lanes(cuda_lib, counts, kind):
    sc = S.dam_break(seed=3, n_side=counts, box=max(counts) * 0.02 + 0.1, **kind)
    a, b = _run(sc, 0), _run(sc, 1)
    for k in a:
        assert np.array_equal(a[k].cpu().numpy(), b[k].cpu().numpy()), k


def test_coupled_solids_do_not_depend_on_the_lanes(cuda_lib):
    sc = S.rigid_drop(seed=2, coupling=2)
    sc.particles.x[sc.particles.phase_id >= 2000, 1] -= 0.05  # into reach of the fluid
    sc.config["Configuration"]["boundaryViscosity"] = 0.5
    a, b = _run(sc, 0), _run(sc, 2)
    for k in a:
        assert np.array_equal(a[k].cpu().numpy(), b[k].cpu().numpy()), k


@pytest.mark.parametrize("counts,kind", [((1, 1, 1), {}), ((9, 7, 8), CROSS), ((21, 20, 19), CROSS), ((26, 25, 24), CROSS),
                                         ((35, 34, 33), CROSS), ((39, 40, 41), CROSS)])
def test_one_kernel_loops_equal_the_host_driven_ones(cuda_lib, counts, kind):
    """The captured step's loops, one cooperative kernel each where the scene splits a
    particle over lanes (and the viscosity's below its own limit), against the separate
    kernels that the host drives: the same fields and iteration counts, over steps in which
    every loop runs several bodies."""
    sc = S.dam_break(seed=5, n_side=counts, box=max(counts) * 0.02 + 0.1, **kind)
    sc.config["Configuration"].update(maxError=0.002, maxErrorV=0.02)
    sc.config["FluidParticles"][0].update(viscoMaxError=1e-6)
    x = sc.particles.x
    nf = sc.particles.n_fluid
    x[:nf] = x[0] + (x[:nf] - x[0]) * 0.92  # above the rest density: the density solve iterates
    out = []
    for host in (False, True):
        m = sph.initialize(SimConfig(config=sc.config), particles=sc.particles)
        solver = sph.build_solver()
        solver.host_loop = host
        solver.initialize()
        g = torch.Generator("cuda").manual_seed(2)
        m.pd.v.copy_((torch.rand(m.pd.v.shape, generator=g, device="cuda") - 0.5) * m.pd.is_dynamic[:, None])
        its = []
        for _ in range(3):
            solver.step()
            st = solver.stats()
            assert st["status"] == 0
            its.append((st["iterations_v"], st["iterations"], st["cg_iterations"]))
        out.append((its, *[getattr(m.pd, k).cpu().numpy() for k in ("x", "v", "acceleration")]))
    assert out[0][0] == out[1][0]
    assert nf < 100 or (max(i[0] for i in out[0][0]) > 0 and max(i[1] for i in out[0][0]) > 1), out[0][0]
    for a, b in zip(out[0][1:], out[1][1:]):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("seed,counts,max_nb", [(1, (1, 1, 1), 64), (2, (3, 5, 7), 64), (3, (13, 13, 13), 64),
                                                (4, (17, 9, 31), 40)])
@pytest.mark.parametrize("cell_factor", [1, 2])
def test_list_build_per_row(cuda_lib, seed, counts, max_nb, cell_factor):
    """Small scenes build their lists one cell row per warp: against brute force, in a
    scene with ragged warps and a crowded cell (windows past the hit mask), under both
    stencils; a too small capacity reports the overflow with the true count."""
    from nonnewton_b200 import _abi

    sc = S.dam_break(seed=seed, n_side=counts, box=max(counts) * 0.02 + 0.04)
    x = sc.particles.x
    crowd = min(90, len(x) // 8)
    x[:crowd] = x[0] + np.random.default_rng(seed).uniform(0, 0.015, (crowd, 3)).astype(np.float32)
    m = sph.initialize(SimConfig(config=sc.config), particles=sc.particles, max_neighbors=256,
                       tuning=dict(cell_factor=cell_factor))
    m.ns.run_search()
    width = 200
    num, lists = m.engine.neighbors(len(x), width)
    xt = m.pd.x
    r = xt[:, None] - xt[None]
    d = (r[..., 0] * r[..., 0] + r[..., 1] * r[..., 1] + r[..., 2] * r[..., 2]).sqrt()
    near = (d < torch.tensor(sc.param.support_radius, dtype=torch.float32, device="cuda"))
    near.fill_diagonal_(False)
    want = torch.full((len(x), width), -1, dtype=torch.int32, device="cuda")
    i, j = near.nonzero(as_tuple=True)
    want[i, torch.arange(len(i), device="cuda") - (near.sum(1).cumsum(0) - near.sum(1))[i]] = j.int()
    assert torch.equal(num, near.sum(1).int()) and torch.equal(lists, want)
    # narrower rows keep the smallest ids
    _, cut = m.engine.neighbors(len(x), 7)
    assert torch.equal(cut, want[:, :7])
    if int(num.max()) > max_nb:
        m.engine.set_neighbor_cap(max_nb)
        m.engine.run_pass(_abi.NN_PASS_SEARCH)
        st = m.engine.stats(0)
        assert st["status"] == _abi.NN_ERR_NEIGHBOR_OVERFLOW and st["max_neighbors_seen"] == int(num.max())


@pytest.mark.parametrize("n_body,coupling", [((4, 4, 4), 1), ((3, 5, 2), 3)])
def test_rigid_substeps_in_one_block(cuda_lib, n_body, coupling):
    """The rigid bodies' substeps run in one block up to a slot capacity, as separate kernels
    above it: a batch of each capacity over the same scene. The sums are FP64 atomics in
    both, so positions agree to the last bits of f32."""
    from nonnewton_b200.batch import Batch

    sc = S.rigid_drop(seed=6, n_body=n_body, coupling=coupling)
    sc.particles.x[sc.particles.phase_id >= 2000, 1] -= 0.05
    out = []
    for capacity in (sc.particles.n, 8193):
        b = Batch(capacity, 1)
        b.set([sc])
        b.step(3)
        assert b.stats(0)["status"] == 0
        out.append(b.scene_view(0, "x").cpu().numpy())
    assert sc.particles.n <= 8192
    assert np.abs(out[0] - out[1]).max() <= 2e-7  # an ulp or two at the domain's size
