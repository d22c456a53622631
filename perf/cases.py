"""The work that a user of this framework has it do, as cases that can be timed.

A case is a dict of plain values; `listed()` names the ones that stand for the ranges and
`draw()` gives more of the same ranges. `prepare()` builds what a program holds before the
call, `run()` makes the call through the public entry points, `work()` says what the call
cannot do without and `exact()` gives the step's results in 64 bits, in plain torch.

Four things are asked of the framework:
  step     one `solver.step()` of a scene through the object API, from particle positions
           and velocities the program sets before it (as a coupled or replayed run does);
  batch    one `Batch.step()` of a set of independent scenes of uneven sizes;
  search   `meta.ns.run_search()` and the neighbour lists it leaves, in particle order;
  surface  `SRTool.dual_contouring` / `marching_cubes` of a particle set.
The scenes are the generators of `nonnewton_b200/scene.py` at the sizes its benchmark,
served workload and tests use. `packing` scales the fluid lattice: 1 is the generators'
starting lattice (about 800 kg/m^3, the free-falling and freshly poured states), 0.93 the
rest density (settled states, in which the pressure solve iterates).
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

from nonnewton_b200 import scene as S
from nonnewton_b200 import sph
from nonnewton_b200.batch import Batch
from nonnewton_b200.config import SimConfig
from nonnewton_b200.surface import SRTool

DEV = "cuda"


def listed():
    return [
        # the smallest scenes of the served range: a splash of 2k fluid particles, where a
        # step is mostly launches and latency (Newtonian, explicit viscosity: the defaults)
        dict(name="step_small_2k", what="step", model="newtonian", side=13, packing=1.0, wiggle=0.02),
        # a rigid body falling into a shallow layer, two coupling substeps: small, with the
        # longest chain of launches
        dict(name="step_rigid_3k", what="step", model="rigid", side=10, packing=1.0, wiggle=0.02),
        # the classic dam break of the benchmark (8,000 fluid in a 15,002-particle box)
        dict(name="step_dam_23k", what="step", model="dam", side=20, packing=1.0, wiggle=0.02),
        # the shear-thinning drop of the benchmark (Cross law, implicit viscosity, CFL)
        dict(name="step_drop_135k", what="step", model="drop", side=50, packing=1.0, wiggle=0.02),
        # a settled pool of the served kind (Cross law, implicit viscosity) at rest density
        dict(name="step_pool_90k", what="step", model="cross", side=41, packing=0.93, wiggle=0.08),
        # the fluid-elastic scene of the benchmark: an elastic block over a pool
        dict(name="step_elastic_176k", what="step", model="elastic", side=40, packing=1.0, wiggle=0.02),
        # a large settled pool: the solver loops iterate on lists longer than a lattice's
        dict(name="step_pool_900k", what="step", model="carreau", side=50, packing=0.93, wiggle=0.08),
        # the benchmark's headline scene (2,000,000 fluid in a 400,002-particle box)
        dict(name="step_carreau_2400k", what="step", model="carreau", side=200, packing=1.0, wiggle=0.02),
        # the served form: scenes of 2k to 128k fluid particles stepped together
        dict(name="batch_mixed_16", what="batch", model="served", side=16, packing=1.0, wiggle=0.02),
        # a program that only wants the neighbour lists of its particles
        dict(name="search_135k", what="search", model="drop", side=50, packing=1.0, wiggle=0.05),
        # the mesh of a small particle ball, as an example or a preview asks for
        dict(name="surface_ball_2k", what="surface", model="ball", side=15, method="dual", normals=True,
             velocity=False),
        # the mesh of the benchmark's drop, frame after frame
        dict(name="surface_drop_125k", what="surface", model="block", side=50, method="dual", normals=True,
             velocity=False),
    ]


def draw(rng):
    def log_int(a, b):
        return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))

    what = rng.choice(("step", "step", "step", "step", "step", "batch", "search", "surface"))
    packing = rng.choice((1.0, 1.0, 0.93))
    wiggle = round(rng.uniform(0.01, 0.04) if packing == 1.0 else rng.uniform(0.03, 0.1), 4)
    if what == "step":
        model = rng.choice(("newtonian", "dam", "drop", "cross", "elastic", "rigid", "carreau"))
        lo, hi = {"newtonian": (13, 50), "dam": (8, 40), "drop": (13, 50), "cross": (13, 50), "elastic": (8, 40),
                  "rigid": (6, 16), "carreau": (20, 200)}[model]
        if model in ("elastic", "rigid"):
            packing, wiggle = 1.0, min(wiggle, 0.04)
        return dict(what=what, model=model, side=log_int(lo, hi), packing=packing, wiggle=wiggle)
    if what == "batch":
        return dict(what=what, model="served", side=log_int(2, 16), packing=packing, wiggle=wiggle)
    if what == "search":
        return dict(what=what, model=rng.choice(("dam", "drop", "cross")), side=log_int(13, 50), packing=packing,
                    wiggle=wiggle)
    return dict(what=what, model=rng.choice(("ball", "block")), side=log_int(8, 50),
                method=rng.choice(("dual", "dual", "cubes")), normals=rng.random() < 0.5,
                velocity=rng.random() < 0.3)


# ---- scenes -------------------------------------------------------------------------
def _half_full(side, r=0.01, **kw):
    """A dam break in a box twice the fluid's volume, as the served requests have it."""
    sp = 2 * r
    edge = max((2.0 * side ** 3) ** (1 / 3), side + 2) * sp
    return S.dam_break(seed=0, n_side=(side,) * 3, box=math.ceil(edge / sp) * sp, r=r, **kw)


@functools.lru_cache(maxsize=4)
def _scenes(model, side):
    """The scenes of a case, with the generators' own jitter seed."""
    if model == "newtonian":
        return [_half_full(side)]
    if model == "cross":
        return [_half_full(side, extra_cfg={"useNonNewtonianModel": True},
                           fluid_cfg={"nonNewtonMethod": "CROSS_", "viscosity0": 5.0, "viscosity_inf": 0.01,
                                      "consistency_index": 1.0, "power_index": 0.7, "viscosityMethod": 13,
                                      "viscoMaxError": 1e-3, "viscoMaxIter": 100})]
    if model == "dam":
        return [S.dam_break(seed=0, n_side=(side,) * 3)]
    if model == "drop":
        return [S.shear_thinning_drop(seed=0, n_side=side)]
    if model == "elastic":
        return [S.fluid_elastic(seed=0, n_el=side)]
    if model == "rigid":
        body = max(4, side // 3)
        return [S.rigid_drop(seed=0, n_fluid=(side, 5, side), n_body=(body,) * 3, box=0.02 * (side + 10), coupling=2)]
    if model == "carreau":
        return [S.roofline_scene(seed=0, counts=(200, max(side // 2, 4), 100))]
    if model == "served":
        rng = np.random.default_rng(1000)
        return [S.served_request(rng) for _ in range(side)]
    raise ValueError(model)


def _flow(sc, case, gen):
    """A mid-simulation state of the scene on the GPU: the fluid lattice at the case's
    packing, each particle moved by `wiggle` spacings, in a smooth divergence-free swirl
    with a little noise; an elastic block is deformed, a rigid body has reached the fluid.
    Returns float32 (x, v)."""
    ps, p = sc.particles, sc.param
    sp = p.particle_diameter
    x = torch.from_numpy(np.ascontiguousarray(ps.x)).to(DEV, torch.float64)
    dyn = torch.from_numpy(ps.is_dynamic).to(DEV).bool()
    phase = torch.from_numpy(ps.phase_id).to(DEV)
    fluid = torch.from_numpy(ps.material).to(DEV) == sph.FLUID
    lo = x[fluid].amin(0)
    gap = 0.5 * sp * (case["packing"] < 1.0)  # settled fluid keeps off the boundary layer
    x[fluid] = lo + gap + (x[fluid] - lo) * case["packing"]
    noise = torch.rand(x.shape, generator=gen, device=DEV, dtype=torch.float64) * 2 - 1
    x += noise * (case["wiggle"] * sp * fluid[:, None])
    rigid = (phase >= 2000) & (phase < 3000)
    x[:, 1] -= 2.0 * sp * rigid
    elastic = phase >= 3000
    if bool(elastic.any()):
        c = x[elastic]
        side = float((c.amax(0) - c.amin(0)).amax())
        x[elastic] = c + 0.01 * side * torch.sin(2 * math.pi * (c[:, [1, 2, 0]] - c.amin(0)) / side + noise[:1])
    k = 2 * math.pi / float(np.max(p.domain_size))
    shift = torch.rand(3, generator=gen, device=DEV, dtype=torch.float64) * 6
    v = 0.4 * (torch.sin(k * x[:, [1, 2, 0]] + shift) + 0.5 * torch.cos(k * x[:, [2, 0, 1]] - shift))
    v += 0.01 * (torch.rand(x.shape, generator=gen, device=DEV, dtype=torch.float64) * 2 - 1)
    v[:, 1] -= 0.5
    v *= dyn[:, None]
    return x.float(), v.float()


def _points(case, seed):
    """A lattice ball or block of particles at 0.02 m, each moved by up to a tenth of the
    spacing, with the bounding box a scene of that size would have; and their velocities."""
    gen = torch.Generator(DEV).manual_seed(int(seed))
    n, sp = case["side"], 0.02
    g = (torch.arange(n, device=DEV, dtype=torch.float64) - (n - 1) / 2) * sp
    x = torch.stack(torch.meshgrid(g, g, g, indexing="ij"), -1).reshape(-1, 3)
    if case["model"] == "ball":
        x = x[x.norm(dim=1) <= (n / 2) * sp]
    box = n * sp + 1.0
    x = x + box / 2
    x += (torch.rand(x.shape, generator=gen, device=DEV, dtype=torch.float64) - 0.5) * 0.2 * sp
    v = torch.sin(3.0 * x[:, [1, 2, 0]])
    return x.float().contiguous(), v.float().contiguous(), box


# ---- the cases ----------------------------------------------------------------------
def prepare(case, seed):
    what = case["what"]
    if what == "surface":
        x, v, box = _points(case, seed)
        sr = SRTool([[0.0] * 3, [box] * 3], voxel_size=0.01, particle_radius=0.02, record_normals=case["normals"],
                    record_velocity=case["velocity"], max_num_vertices=40 * len(x) + 20000,
                    max_num_indices=200 * len(x) + 100000, max_num_particles=len(x))
        # the program's own mesh buffers (as a renderer keeps them), which each frame's mesh fills
        nv = 30 * case["side"] ** 2 * (5 if case["method"] == "cubes" else 1) + 4000
        f = dict(dtype=torch.float32, device=DEV)
        buf = dict(vertex=torch.zeros(nv, 3, **f), index=torch.zeros(6 * nv, dtype=torch.int32, device=DEV),
                   normal=torch.zeros(nv, 3, **f), velocity=torch.zeros(nv, 3, **f))
        return dict(case=case, sr=sr, x=x, v=v, buf=buf)
    gen = torch.Generator(DEV).manual_seed(int(seed))
    scenes = _scenes(case["model"], case["side"])
    if what == "batch":
        n = sum(sc.particles.n for sc in scenes)
        batch = Batch(n, len(scenes))
        batch.set(scenes)
        flows = [_flow(sc, case, gen) for sc in scenes]
        return dict(case=case, batch=batch, x=torch.cat([f[0] for f in flows]), v=torch.cat([f[1] for f in flows]),
                    fluid=batch.pd.material[:n] == sph.FLUID)
    sc = scenes[0]
    sph.initialize(SimConfig(config=sc.config), particles=sc.particles, quirks=sc.param.quirks)
    solver = sph.build_solver()
    solver.initialize()
    x, v = _flow(sc, case, gen)
    # `meta` is the object API's global: a program with several simulations keeps each one's
    return dict(case=case, meta=dict(vars(sph.meta)), pd=sph.meta.pd, ns=sph.meta.ns, solver=solver, x=x, v=v,
                nf=sc.particles.n_fluid)


def run(state):
    case = state["case"]
    what = case["what"]
    if what == "surface":
        sr = state["sr"]
        entry = sr.dual_contouring if case["method"] == "dual" else sr.marching_cubes
        entry(0.0, 0.06, len(state["x"]), state["x"], velocity=state["v"] if case["velocity"] else None)
        mesh = dict(vertex=sr.mesh_vertex, index=sr.mesh_index, normal=sr.mesh_normal, velocity=sr.mesh_velocity)
        for k, t in mesh.items():
            if len(t):
                state["buf"][k][:len(t)].copy_(t)
        out = {k: state["buf"][k] for k, t in mesh.items() if len(t)}
        return dict(out, vertices=int(sr.num_vertices), indices=int(sr.num_indices))
    if what == "batch":
        batch = state["batch"]
        n = batch.n
        batch.pd.x[:n].copy_(state["x"])
        batch.pd.v[:n].copy_(state["v"])
        batch.step(1)
        return _fields(batch.pd, n, state["fluid"], True, False)
    vars(sph.meta).update(state["meta"])
    pd = state["pd"]
    pd.x.copy_(state["x"])
    if what == "search":
        ns = state["ns"]
        ns.run_search()
        return dict(num=ns.num_neighbors, lists=ns.neighbors)
    pd.v.copy_(state["v"])
    state["solver"].step()
    return _fields(pd, pd.particle_max_num, slice(0, state["nf"]),
                   case["model"] in ("drop", "cross", "elastic", "carreau"), case["model"] == "elastic")


def _fields(pd, n, fluid, nonnewton, elastic):
    """The particle fields a step writes (the solver's own ones for fluid particles)."""
    out = dict(x=pd.x[:n], v=pd.v[:n], a=pd.acceleration[:n], volume=pd.volume[:n], density=pd.density[:n],
               factor=pd.dfsph_factor[:n][fluid], density_adv=pd.density_adv[:n][fluid])
    if nonnewton:
        out.update(strain_rate=pd.strain_rate_norm[:n], viscosity=pd.nonnewton_viscosity[:n])
    if elastic:
        el = pd.phase_id[:n] >= 3000
        out.update(stress=pd.stress[:n][el], rotation=pd.rotations[:n][el])
    return out


def work(case):
    """Inputs read once and outputs written once; arithmetic at 30 neighbours a particle."""
    if case["what"] == "surface":
        n = case["side"] ** 3 * (math.pi / 6 if case["model"] == "ball" else 1.0)
        area = 6 * (2 * case["side"]) ** 2  # mesh vertices: about one per crossed voxel
        per_v = 12 + 24 + 12 * case["normals"] + 12 * case["velocity"]
        inside = 4 / 3 * math.pi * (0.12 / 0.01) ** 3  # vertices a particle's kernel reaches
        return dict(bytes=n * (12 + 12 * case["velocity"]) + area * per_v, flops=n * inside * 20)
    scenes = _scenes(case["model"], case["side"])
    n = sum(sc.particles.n for sc in scenes)
    nf = sum(sc.particles.n_fluid for sc in scenes)
    if case["what"] == "search":  # positions in, 60-wide id lists and counts out
        return dict(bytes=n * (12 + 4 + 240), flops=n * 30 * 8)
    # x, v, volume, mass, density, three class fields in; x, v, a and four scalars out
    implicit = scenes[0].param.implicit_viscosity
    passes = 10 if implicit else 8
    return dict(bytes=n * (48 + 52) + nf * 8, flops=nf * 30 * 25 * passes)


# ---- the step in 64 bits ------------------------------------------------------------
def _pairs(x, h):
    """All (i, j), i != j, with |x_i - x_j| < h as 32-bit arithmetic rounds it, the rule
    of the search; sorted by i."""
    h32 = torch.tensor(h, dtype=torch.float32, device=x.device)
    n = len(x)
    c = torch.floor((x.double() - x.double().amin(0)) / (h * 1.001)).long() + 1
    d = c.amax(0) + 2
    key = (c[:, 0] * d[1] + c[:, 1]) * d[2] + c[:, 2]
    keys, order = torch.sort(key)
    ii, jj = [], []
    for dx in (-1, 0, 1):
        for dy in (-1, 0, 1):
            at = key + (dx * d[1] + dy) * d[2]
            b = torch.searchsorted(keys, at - 1)
            cnt = torch.searchsorted(keys, at + 1, right=True) - b
            i = torch.repeat_interleave(torch.arange(n, device=x.device), cnt)
            first = torch.cumsum(cnt, 0) - cnt
            j = order[b[i] + torch.arange(len(i), device=x.device) - first[i]]
            r = x[i] - x[j]
            q = r * r
            near = (((q[:, 0] + q[:, 1]) + q[:, 2]).sqrt() < h32) & (i != j)
            ii.append(i[near])
            jj.append(j[near])
    i, j = torch.cat(ii), torch.cat(jj)
    o = torch.argsort(i, stable=True)
    return i[o], j[o]


def _cubic(r, h):
    """(W, grad W) of the cubic spline at the pair offsets r."""
    rn = r.norm(dim=1)
    q = (rn / h).clamp(max=1.0)
    k = 8.0 / math.pi / h ** 3
    t = 1 - q
    w = torch.where(q <= 0.5, k * (6 * q * q * (q - 1) + 1), 2 * k * t ** 3)
    f = torch.where(q <= 0.5, 6 * k * q * (3 * q - 2), -6 * k * t * t)
    g = torch.where((rn > 1e-5)[:, None], r / (rn * h)[:, None], torch.zeros_like(r)) * f[:, None]
    return w, g


def _law(p, g):
    if p.nonnewton_method == 2:  # Cross
        return p.viscosity_inf + (p.viscosity0 - p.viscosity_inf) / (1 + (p.consistency_index * g) ** p.power_index)
    if p.nonnewton_method == 4:  # Carreau, in the reference's form
        return p.viscosity_inf + (p.viscosity0 - p.viscosity_inf) / (
            1 + (p.consistency_index * g * g) ** ((1 - p.power_index) / 2))
    raise NotImplementedError(p.nonnewton_method)


def _rotation(A):
    U, _, Vt = torch.linalg.svd(A)
    s = torch.det(U @ Vt).sign()
    U = torch.cat([U[:, :, :2], U[:, :, 2:] * s[:, None, None]], 2)
    return U @ Vt


def _step64(sc, x32, v32):
    """One step of the scene from (x, v) in float64; the fields of `_fields`."""
    p, ps = sc.param, sc.particles
    h, sp, rho0 = p.support_radius, p.particle_diameter, p.density0
    dev = x32.device
    f64 = dict(dtype=torch.float64, device=dev)
    x, v = x32.double(), v32.double()
    rest = torch.from_numpy(np.ascontiguousarray(ps.x, dtype=np.float32)).to(dev)
    m = torch.from_numpy(ps.mass.astype(np.float32)).to(**f64)
    fluid = torch.from_numpy(ps.material).to(dev) == sph.FLUID
    dyn = torch.from_numpy(ps.is_dynamic).to(dev).bool()
    phase = torch.from_numpy(ps.phase_id).to(dev)
    n, nf = len(x), ps.n_fluid
    k_w = 8.0 / math.pi / h ** 3
    i, j = _pairs(x32, h)
    r = x[i] - x[j]
    W, gW = _cubic(r, h)

    def gather(val, at=i):  # sum of a per-pair value over each particle's neighbours
        return torch.zeros((n,) + val.shape[1:], **f64).index_add_(0, at, val)

    dt = p.dt
    if p.cfl:
        vm = float(v32[dyn].norm(dim=1).max())
        if vm > 1e-9:
            dt = p.cfl_factor * 0.4 * sp / vm
        dt = min(max(dt, p.cfl_min_dt), p.cfl_max_dt)
    # boundary volumes: of static solids at the initial positions, of moving ones now
    V = torch.full((n,), p.volume0, **f64)
    i0, j0 = _pairs(rest, h)
    ss = ~fluid[i0] & ~fluid[j0]
    w0, _ = _cubic((rest.double()[i0] - rest.double()[j0])[ss], h)
    static = ~fluid & ~dyn
    V = torch.where(static, 3.0 / (k_w + gather(w0, i0[ss])), V)
    V = torch.where(~fluid & dyn, 3.0 / (k_w + gather(W * ~fluid[j])), V)
    g = torch.tensor(np.asarray(p.gravity), **f64)
    a = torch.where(static[:, None], torch.zeros(n, 3, **f64), g.expand(n, 3)).clone()
    # the pairs of fluid particles, which the solvers walk
    keep = fluid[i]
    fi, fj = i[keep], j[keep]
    r, W, gW = r[keep], W[keep], gW[keep]
    to_fluid = fluid[fj]
    count = torch.zeros(n, dtype=torch.long, device=dev).index_add_(0, fi, torch.ones_like(fi))
    density = torch.from_numpy(np.full(n, rho0, np.float32)).to(**f64)
    density = torch.where(fluid, rho0 * (V * k_w + gather(V[fj] * W, fi)), density)
    G = V[fj, None] * gW
    total = gather(((G * G).sum(1)) * to_fluid, fi) + (gather(G, fi) ** 2).sum(1)
    alpha = torch.where(total > 1e-6, -1.0 / total.clamp(min=1e-30), torch.zeros_like(total)) * fluid

    def change():
        dd = gather(((v[fi] - v[fj]) * G).sum(1), fi).clamp(min=0)
        return torch.where(count < 20, torch.zeros_like(dd), dd) * fluid

    def push(kappa):  # the velocity change that a solver iteration makes
        ks = kappa[fi] + torch.where(to_fluid, kappa[fj], torch.zeros_like(kappa[fj]))
        ks = torch.where(ks.abs() > p.m_eps, ks, torch.zeros_like(ks))
        return gather(G * (dt * ks)[:, None], fi)

    adv = change()
    alpha = alpha / dt
    it = 0
    while True:
        v = v + push(adv * alpha)
        adv = change()
        if float(rho0 * adv.sum()) / nf <= 1.0 / dt * p.max_error_v * 0.01 * rho0:
            break
        it += 1
        if it >= max(p.max_iterations_v, 1):
            break
    alpha = alpha * dt
    # forces other than the pressure
    r2 = (r * r).sum(1)
    vij = v[fi] - v[fj]
    c01 = 0.01 * h * h
    if p.use_surface_tension:
        w_d = float(_cubic(torch.tensor([[sp, 0.0, 0.0]], **f64), h)[0][0])
        st = -(p.surface_tension / m[fi] * m[fj] * torch.where(r2 > sp * sp, W, torch.full_like(W, w_d)) * to_fluid)
        a += gather(st[:, None] * r, fi)
    srn, mu = torch.zeros(n, **f64), torch.full((n,), p.viscosity * rho0, **f64)
    if p.use_nonnewtonian:
        D = -(vij[:, :, None] * gW[:, None, :]) * m[fj, None, None]
        D = gather((D + D.transpose(1, 2)).reshape(-1, 9), fi) * (0.5 / density)[:, None]
        srn = D.norm(dim=1) * fluid
        mu = torch.where(fluid, _law(p, srn), torch.zeros_like(srn))
    if p.implicit_viscosity:
        vol = m / density
        c = dt * 10 * 0.5 * (mu[fi] + mu[fj]) * vol[fi] * vol[fj] / (r2 + c01) * to_fluid

        def A(y):
            return m[:, None] * y - gather(gW * (c * (r * (y[fi] - y[fj])).sum(1))[:, None], fi)

        blocks = torch.eye(3, **f64) * m[:, None, None]
        blocks = blocks - gather((gW[:, :, None] * r[:, None, :] * c[:, None, None]).reshape(-1, 9), fi).reshape(-1, 3, 3)
        inverse = torch.linalg.inv(blocks)
        on = fluid[:, None]
        y, b = v * on, m[:, None] * v * on
        res = (b - A(y)) * on
        z = (inverse @ res[:, :, None])[:, :, 0]
        d, rz, bb = z, (res * z).sum(), float((b * b).sum())
        rel = math.sqrt(float((res * res).sum()) / bb) if bb > 0 else 0.0
        it = 0
        while rel > p.visco_max_error and it < p.visco_max_iter:
            Ad = A(d) * on
            al = rz / (d * Ad).sum()
            y, res = y + al * d, res - al * Ad
            z = (inverse @ res[:, :, None])[:, :, 0]
            rz, old = (res * z).sum(), rz
            it += 1
            rel = math.sqrt(float((res * res).sum()) / bb)
            d = z + rz / old * d
        a = a + torch.where(on, (y - v) / dt, torch.zeros_like(v))
    elif p.use_viscosity:
        f = 10 * p.viscosity * m[fj] / density[fj] * (vij * r).sum(1) / (r2 + c01) * to_fluid
        a += gather(gW * f[:, None], fi)
    v = torch.where((fluid & dyn)[:, None], v + dt * a, v)
    # pressure
    def advected():
        d = density / rho0 + dt * gather(((v[fi] - v[fj]) * G).sum(1), fi)
        return torch.where(fluid, d.clamp(min=1.0), torch.ones_like(d))

    adv = advected()
    alpha = alpha / (dt * dt)
    moving = ~fluid & dyn
    couple = moving[i] & fluid[j]
    si, sj = i[couple], j[couple]
    gS = _cubic(x[si] - x[sj], h)[1]
    it = 0
    while True:
        kappa = (adv - 1) * alpha
        ks = torch.where(kappa[sj].abs() > p.m_eps, kappa[sj], torch.zeros_like(kappa[sj]))
        a = a + gather(gS * (V[si] * ks)[:, None], si)
        v = v + push(kappa)
        adv = advected()
        if float(rho0 * (adv - 1).sum()) / nf <= p.max_error * 0.01 * rho0:
            break
        it += 1
        if it >= max(p.max_iterations, 1):
            break
    out = dict(volume=V, density=density, factor=alpha[:nf], density_adv=adv[:nf])
    if p.use_nonnewtonian:
        out.update(strain_rate=srn, viscosity=mu)
    if p.has_elastic:
        el = phase >= 3000
        both = el[i0] & el[j0] & (phase[i0] == phase[j0])
        ei, ej = i0[both], j0[both]
        r0 = rest.double()[ej] - rest.double()[ei]
        w, gw = _cubic(r0, h)
        v0 = m / (m * k_w + gather(m[ej] * w, ei))
        rc = x[ej] - x[ei]
        F = gather((rc[:, :, None] * r0[:, None, :]).reshape(-1, 9) * (m[ei] * w)[:, None], ei).reshape(-1, 3, 3)
        R = torch.eye(3, **f64).repeat(n, 1, 1)
        R[el] = _rotation(F[el])
        u = ((R[ei].transpose(1, 2) @ rc[:, :, None])[:, :, 0] - r0) * v0[ej, None]
        Gr = -gather((u[:, :, None] * gw[:, None, :]).reshape(-1, 9), ei).reshape(-1, 3, 3)
        E = 0.5 * (Gr + Gr.transpose(1, 2))
        lam = p.youngs_modulus / ((1 + p.poisson_ratio) * (1 - 2 * p.poisson_ratio))
        cd, co, cs = lam * (1 - p.poisson_ratio), lam * p.poisson_ratio, lam * 0.5 * (1 - 2 * p.poisson_ratio)
        tr = E.diagonal(dim1=1, dim2=2).sum(1)
        eye = torch.eye(3, **f64)
        T = torch.where(eye.bool(), (cd - co) * E + co * tr[:, None, None], cs * E)
        vv = (v0[ei] * v0[ej])[:, None]
        fij = -(T[ej] @ gw[:, :, None])[:, :, 0] * vv
        fji = (T[ei] @ gw[:, :, None])[:, :, 0] * vv
        f = (R[ej] @ fij[:, :, None])[:, :, 0] - (R[ei] @ fji[:, :, None])[:, :, 0]
        a = a + torch.where(el[:, None], 0.5 * gather(f, ei) / m[:, None], torch.zeros_like(a))
        T6 = torch.stack([T[:, 0, 0], T[:, 1, 1], T[:, 2, 2], T[:, 0, 1], T[:, 0, 2], T[:, 1, 2]], 1)
        out.update(stress=T6[el], rotation=R.reshape(n, 9)[el])
    for body in torch.unique(phase[(phase >= 2000) & (phase < 3000)]).tolist():
        at = phase == body
        q = rest.double()[at]
        q = q - q.mean(0)
        for _ in range(p.coupling_interval):
            x[:, 1] = torch.where(~fluid & (x[:, 1] < p.padding), torch.full_like(x[:, 1], p.padding), x[:, 1])
            cm = x[at].mean(0)
            R = _rotation(torch.einsum("ni,nj->ij", x[at] - cm, q)[None])[0]
            x[at] = cm + q @ R.T
    # advection and the domain walls
    v = torch.where(moving[:, None], v + dt * a, v)
    x = torch.where(dyn[:, None], x + dt * v, x)
    lo = torch.tensor(p.domain_start + p.padding, **f64)
    hi = torch.tensor(p.domain_end - p.padding, **f64)
    normal = ((x > hi).double() - (x <= lo).double()) * dyn[:, None]
    hit = normal.norm(dim=1, keepdim=True)
    unit = normal / hit.clamp(min=1e-6)
    bounced = (v - unit * ((1 + p.collision_coeff) * (v * unit).sum(1, keepdim=True))) * p.sticky_coeff
    v = torch.where(hit > 0, bounced, v)
    x = torch.where(dyn[:, None], torch.minimum(torch.maximum(x, lo), hi), x)
    return dict(out, x=x, v=v, a=a)


def exact(case, seed):
    """The step's fields in 64 bits. None for the searches (whole numbers) and for the
    surfaces, whose mesh hangs on comparisons that are made in 32 bits by definition."""
    if case["what"] not in ("step", "batch"):
        return None
    gen = torch.Generator(DEV).manual_seed(int(seed))
    scenes = _scenes(case["model"], case["side"])
    flows = [_flow(sc, case, gen) for sc in scenes]
    outs = [_step64(sc, *f) for sc, f in zip(scenes, flows)]
    return {k: torch.cat([o[k] for o in outs]) for k in outs[0]}
