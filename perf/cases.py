"""The work that users of this framework have it do, as measurable cases.

A case is one pass through the public entry points on a state that a user's
program would hold: a coupled WCSPH-DEM step of a running dam break, one step
of a batched ensemble, an SPH-only step, a DEM-only step, the single coupling
kernels, the surrogate's graph and inference, and one training step.

States are made from the seed: the generator's scene with the disorder a
running simulation has (lattice positions moved by a few percent of dx, a
smooth flow field plus noise, densities a fraction of a percent off rest) and
spheres straddling or inside the water.  ``exact`` restates the step, the
contacts, the coupling and the network in plain torch with 64-bit numbers.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

from warp_sph_gpt_gb300 import HashGrid, SPHDEM_OneStep, dem_search_scales, kernels
from warp_sph_gpt_gb300.batch import Ensemble
from warp_sph_gpt_gb300.generate import (CoupledGenerationConfig, DEMPtlGeneration, build_case, config_batch_member,
                                         config_large, solver_config)
from warp_sph_gpt_gb300.simulation import run_steps
from warp_sph_gpt_gb300.surrogate import Graph, Network, Sets, SurrogateConfig, prepare_target

DEV = "cuda"
SEARCH_PAIRS_MAX = 3.0e9  # pairs beyond which the 64-bit restatement takes too long


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # the reference's own example (config 1), one call of the step API per
        # step as its main loop does: the smallest call, latency and launches
        dict(name="step_small", kind="step", scene="tank", dx=0.02, fx=25, fy=20, fz=25, tx=100, ty=20, tz=50,
             dem=(5 * 10000 + 2 * 100 + 2), z0=0.42, steps=1),
        # the 100k-particle tank with its 160 spheres in the water, where the
        # porosity of nearly every particle has to be found
        dict(name="step_submerged_100k", kind="step", scene="tank", dx=0.01, fx=50, fy=40, fz=50, tx=200, ty=40,
             tz=100, dem=(10 * 10000 + 4 * 100 + 4), z0=0.16, steps=1),
        # the same tank early in the run: the spheres meet the surface
        dict(name="step_surface_100k", kind="step", scene="tank", dx=0.01, fx=50, fy=40, fz=50, tx=200, ty=40,
             tz=100, dem=(10 * 10000 + 4 * 100 + 4), z0=0.46, steps=2),
        # the benchmark's default workload: 792k fluid, 2.2M wall, 2,000 spheres
        # of unequal radii
        dict(name="step_large_800k", kind="step", scene="large", width=0.167, dem=2000, steps=1),
        # an ensemble of 64 uneven dam breaks advanced as one batched state
        dict(name="ensemble_64", kind="ensemble", members=64, first=0, steps=1),
        # WCSPH without spheres, at an odd size
        dict(name="sph_only_47k", kind="sph", scene="tank", dx=0.0125, fx=41, fy=31, fz=37, tx=161, ty=31, tz=81,
             dem=0, z0=0.0, steps=1),
        # a DEM-only step: contacts with their history, walls, integration
        dict(name="dem_only_2000", kind="dem", nx=20, ny=10, nz=10, radius=0.025),
        # the single coupling kernels under the reference's kernel names
        dict(name="coupling_kernels_37k", kind="coupling", scene="tank", dx=0.014, fx=40, fy=28, fz=33, tx=142, ty=28,
             tz=71, dem=(6 * 10000 + 4 * 100 + 4), z0=0.2, steps=1),
        # the density and force kernels under the reference's kernel names
        dict(name="sph_kernels_100k", kind="kernels", scene="tank", dx=0.01, fx=50, fy=40, fz=50, tx=200, ty=40,
             tz=100, dem=0, z0=0.0, steps=1),
        # the surrogate's inference in a rollout: node inputs, radius graph, network
        dict(name="surrogate_infer", kind="infer", member=0, z0=0.42, config1=True),
        # one training iteration on one member's graph
        dict(name="surrogate_train", kind="train", member=5, z0=0.3, config1=False),
        # the same for a small member, where latency and launches count
        dict(name="surrogate_train_small", kind="train", member=-1, z0=0.2, config1=False),
    ]


def draw(rng):
    kind = rng.choice(["step", "step", "ensemble", "sph", "dem", "coupling", "kernels", "infer", "train"])
    if kind == "step" and rng.random() < 0.25:
        return dict(kind="step", scene="large", width=round(math.exp(rng.uniform(math.log(0.03), math.log(0.16))), 3),
                    dem=int(math.exp(rng.uniform(math.log(300), math.log(2000)))), steps=1)
    if kind in ("step", "sph", "coupling", "kernels"):
        dx = round(math.exp(rng.uniform(math.log(0.01), math.log(0.025))), 4)
        ty = max(8, int(rng.uniform(0.2, 0.4) / dx))
        fx, fz = int(rng.uniform(0.25, 0.6) / dx), int(rng.uniform(0.25, 0.5) / dx)
        tx, tz = max(fx + 5, int(rng.uniform(1.0, 2.0) / dx)), max(fz + 10, int(rng.uniform(0.7, 1.0) / dx))
        ny = max(1, int((ty * dx - 0.1) / 0.065))
        dem = rng.randint(1, 9) * 10000 + rng.randint(1, ny) * 100 + rng.randint(1, 4)
        z0 = round(rng.uniform(0.08, fz * dx + 0.05), 3)
        coupled = kind in ("step", "coupling")
        return dict(kind=kind, scene="tank", dx=dx, fx=fx, fy=ty, fz=fz, tx=tx, ty=ty, tz=tz,
                    dem=dem if coupled else 0, z0=z0 if coupled else 0.0,
                    steps=1 if kind in ("coupling", "kernels") else rng.choice((1, 1, 2)))
    if kind == "ensemble":
        return dict(kind="ensemble", members=int(math.exp(rng.uniform(math.log(2), math.log(48)))),
                    first=rng.randint(1, 400), steps=rng.randint(1, 2))
    if kind == "dem":
        return dict(kind="dem", nx=rng.randint(2, 22), ny=rng.randint(2, 10), nz=rng.randint(2, 9),
                    radius=round(rng.uniform(0.012, 0.03), 4))
    return dict(kind=kind, member=rng.randint(0, 400), z0=round(rng.uniform(0.15, 0.5), 3),
                config1=kind == "infer" and rng.random() < 0.3)


# ---------------------------------------------------------------------------
# scenes
# ---------------------------------------------------------------------------
def _gen(case):
    """Generation config, sphere centres and radii of a case's scene (no disorder yet)."""
    if case.get("scene") == "large":
        return config_large(case["width"], seed=3, n_dem=case["dem"])
    dx = case["dx"]
    dem = case["dem"] or 10101
    nx, ny, nz = dem // 10000, dem // 100 % 100, dem % 100
    dt = min(1.0e-4, 0.5e-4 * dx / 0.01)
    gen = CoupledGenerationConfig(
        device="cpu", dx=dx, h=1.3 * dx, dt=dt, tank_width=case["tx"] * dx, tank_depth=case["ty"] * dx,
        tank_height=case["tz"] * dx, fluid_width=case["fx"] * dx, fluid_depth=case["fy"] * dx,
        fluid_height=case["fz"] * dx, dem_nx=nx, dem_ny=ny, dem_nz=nz, dem_origin_x=0.06,
        dem_origin_y=0.5 * (case["ty"] * dx - 0.065 * (ny - 1)), dem_origin_z=case["z0"] or 0.3,
        dem_bnd_radius=0.5 * dx, dem_bnd_spacing=dx)
    pos = DEMPtlGeneration(gen).dem_particle()
    return gen, (pos if case["dem"] else np.zeros((0, 3))), (None if case["dem"] else np.zeros(0))


@functools.lru_cache(maxsize=2)
def _scene(items):
    """Undisturbed structs of a scene on the host, kept so that further seeds need only the disorder."""
    gen, pos, rad = _gen(dict(items))
    return gen, build_case(gen, pos, rad, device="cpu")


def _fresh_scene(case):
    key = ("scene", "dx", "fx", "fy", "fz", "tx", "ty", "tz", "dem", "z0", "width")
    gen, parts = _scene(tuple((k, case[k]) for k in key if k in case))
    return gen, [p.to(DEV) for p in parts]


def _disorder(P, B, D, dx, rho0, seed, lo=None, hi=None):
    """The state a running dam break is in, made in place from the seed."""
    g = torch.Generator(device=DEV).manual_seed(int(seed))
    rand = lambda *s: torch.rand(*s, device=DEV, generator=g)  # noqa: E731
    n = P.n
    P.pos.add_((rand(n, 3) - 0.5) * (0.04 * dx))
    k = 2.0 * math.pi / 0.6
    ph = rand(3) * 2.0 * math.pi
    x, y, z = P.pos[:, 0], P.pos[:, 1], P.pos[:, 2]
    u = torch.stack([0.4 * torch.cos(k * z + ph[0]) * torch.sin(0.5 * k * x + ph[1]) + 0.3,
                     0.05 * torch.sin(k * y + ph[2]), -0.3 * torch.sin(k * x + ph[1])], 1)
    P.vel.copy_(u + 0.02 * (rand(n, 3) - 0.5))
    P.rho.copy_(rho0 * (1.0 + 0.004 * (rand(n) - 0.5)))
    P.flt.copy_(1.0 + 0.01 * (rand(n) - 0.5))
    B.rho.copy_(rho0 * (1.0 + 0.01 * (rand(B.n) - 0.5)))
    if D.n:
        D.pos.add_((rand(D.n, 3) - 0.5) * 0.01)
        D.vel.copy_(0.5 * (rand(D.n, 3) - 0.5) + torch.tensor([0.1, 0.0, -0.4], device=DEV))
        D.omega.copy_(4.0 * (rand(D.n, 3) - 0.5))


class _State:
    pass


def _grids(s, solv, scales):
    s.grids = [HashGrid() for _ in range(4)]
    radii = (solv.support, solv.support, max(2.0 * scales[0], 2.0 * scales[2]), max(2.0 * scales[1], solv.support))
    for g, p, r in zip(s.grids, (s.P, s.B, s.D, s.W), radii):
        g.build(p.pos, r)


def prepare(case, seed):
    s = _State()
    s.case, s.kind, s.step = case, case["kind"], 0
    if s.kind == "ensemble":
        s.E = Ensemble([config_batch_member(case["first"] + i) for i in range(case["members"])], device=DEV)
        s.P, s.B, s.D, s.W, s.solv, s.scales = s.E.P, s.E.B, s.E.D, s.E.W, s.E.solv, s.E.scales
        s.D.pos[:, 2] -= 0.12  # the lowest spheres touch the water
        _disorder(s.P, s.B, s.D, 0.02, s.solv.rho0, seed)
        return s
    if s.kind == "dem":
        return _prepare_dem(s, case, seed)
    if s.kind in ("infer", "train"):
        return _prepare_network(s, case, seed)
    gen, (s.P, s.B, s.D, s.W) = _fresh_scene(case)
    s.solv = solver_config(gen)
    _disorder(s.P, s.B, s.D, gen.dx, gen.rho0, seed)
    s.scales = dem_search_scales(s.D, s.W) if s.D.n else (0.0, gen.dem_bnd_radius, 0.0, 0.0)
    _grids(s, s.solv, (s.scales[0] or 0.05, s.scales[1], s.scales[2] or gen.dem_h))
    if s.kind in ("coupling", "kernels"):  # fields that the single kernels read
        g = torch.Generator(device=DEV).manual_seed(int(seed) + 77)
        rand = lambda *a: torch.rand(*a, device=DEV, generator=g)  # noqa: E731
        s.P.pres.copy_(4.0e3 * rand(s.P.n))
        s.B.pres.copy_(4.0e3 * rand(s.B.n))
        s.P.porosity.copy_(0.6 + 0.4 * rand(s.P.n))
        s.P.acc.copy_(20.0 * (rand(s.P.n, 3) - 0.5))
    return s


def _prepare_dem(s, case, seed):
    """A loose packing that touches its neighbours and the floor and side walls."""
    nx, ny, nz, r = case["nx"], case["ny"], case["nz"], case["radius"]
    sp = 2.0 * r
    dx = 0.02
    up = lambda v: math.ceil((v + 1e-9) / dx) * dx  # noqa: E731
    gen = CoupledGenerationConfig(device="cpu", dx=dx, tank_width=up(nx * sp + 0.2), tank_depth=up(ny * sp),
                                  tank_height=up(nz * sp + 0.3), fluid_width=0.1, fluid_depth=0.1, fluid_height=0.1,
                                  dem_radius=r, dt=2.5e-5)
    k = np.stack(np.meshgrid(np.arange(nx), np.arange(ny), np.arange(nz), indexing="ij"), -1).reshape(-1, 3)
    rng = np.random.default_rng(seed)
    rad = r * rng.uniform(0.96, 1.0, len(k))
    pos = r * 0.985 + k * (sp * 0.985) + rng.uniform(-0.01, 0.01, (len(k), 3)) * r
    s.D, s.W = DEMPtlGeneration(gen).build(DEV, pos, rad)
    s.D.vel.copy_(torch.tensor(rng.normal(0.0, 0.05, (len(k), 3)), dtype=torch.float32))
    s.D.omega.copy_(torch.tensor(rng.normal(0.0, 1.0, (len(k), 3)), dtype=torch.float32))
    s.gen = gen
    s.r_max, s.rb_max = float(s.D.radius.max()), gen.dem_bnd_radius
    s.grids = [HashGrid(), HashGrid()]
    s.grids[1].build(s.W.pos, 2.0 * max(s.r_max, s.rb_max))
    return s


def _member(case):
    if case["config1"]:
        return CoupledGenerationConfig(device="cpu", h=0.026), None, None
    if case["member"] < 0:
        return CoupledGenerationConfig(device="cpu", h=0.026, tank_width=0.8, fluid_width=0.2, fluid_height=0.2,
                                       dem_nx=2), None, None
    return config_batch_member(case["member"])


def _prepare_network(s, case, seed):
    gen, pos, rad = _member(case)
    s.P, s.B, s.D, s.W = build_case(gen, pos, rad, device=DEV)
    if s.D.n:  # down into the water
        s.D.pos[:, 2] += max(0.05, case["z0"]) - s.D.pos[:, 2].min()
    _disorder(s.P, s.B, s.D, gen.dx, gen.rho0, seed)
    g = torch.Generator(device=DEV).manual_seed(int(seed) + 5)
    for part in (s.P, s.D):
        part.acc.copy_(12.0 * (torch.rand(part.n, 3, device=DEV, generator=g) - 0.5))
    s.P.porosity.copy_(0.7 + 0.3 * torch.rand(s.P.n, device=DEV, generator=g))
    s.cfg = SurrogateConfig(radius=0.04, dt=1.0e-4, rho0=1000.0, scale=(2e-5, 4e-2, 1e-6, 2e-3))
    s.net = Network(s.cfg, DEV, seed=int(seed) % 1000)
    s.net.theta[37376:37376 + 768] *= 10.0  # an output layer of the size a trained one has
    s.net.pack()
    s.graph = Graph(s.cfg, DEV)
    s.sets = Sets(s.P, s.B, s.D, s.W)
    s.graph.set_nodes(s.sets)
    s.graph.build()  # grid geometry and edge capacity, once per program
    n = s.P.n + s.D.n
    x, v = torch.cat([s.P.pos, s.D.pos]), torch.cat([s.P.vel, s.D.vel])
    a = torch.cat([s.P.acc, s.D.acc])
    sx = torch.full((n, 1), s.cfg.scale[0], device=DEV)
    sv = torch.full((n, 1), s.cfg.scale[1], device=DEV)
    sx[s.P.n:], sv[s.P.n:] = s.cfg.scale[2], s.cfg.scale[3]
    m, dt = s.cfg.substeps, s.cfg.dt
    s.x_t = x + m * dt * v + 0.5 * dt * dt * m * (m + 1) * a + sx * torch.randn(n, 3, device=DEV, generator=g)
    s.v_t = v + m * dt * a + sv * torch.randn(n, 3, device=DEV, generator=g)
    return s


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
_FLUID = ("rho", "pres", "acc", "vel", "pos")
_COUPLED = _FLUID + ("porosity", "pgf", "acc_dem")
_DEM = ("force", "torque", "vel", "pos", "omega", "drag", "pressure_force", "flt_s", "porosity")


def _outputs(s, fluid, dem=()):
    out = {"P_" + k: getattr(s.P, k) for k in fluid}
    out["B_rho"], out["B_pres"] = s.B.rho, s.B.pres
    out.update({"D_" + k: getattr(s.D, k) for k in dem})
    if dem:
        out["dem_offset"], out["bnd_offset"] = s.D.contact_dem_offset_old, s.D.contact_bnd_offset_old
    return out


def run(s):
    kind = s.kind
    if kind == "step":
        n = s.case["steps"]
        if n == 1:
            SPHDEM_OneStep(s.solv, s.P, s.B, s.D, s.W, *s.grids, s.step, s.scales)
        else:
            run_steps(s.solv, s.P, s.B, s.grids[0], s.grids[1], s.D, s.W, s.grids[2], s.grids[3], first_step=s.step,
                      n_steps=n, search_scales=s.scales)
        s.step += n
        return _outputs(s, _COUPLED, _DEM)
    if kind == "ensemble":
        s.E.run(s.step, s.case["steps"])
        s.step += s.case["steps"]
        return _outputs(s, _COUPLED, _DEM)
    if kind == "sph":
        run_steps(s.solv, s.P, s.B, s.grids[0], s.grids[1], first_step=s.step, n_steps=s.case["steps"])
        s.step += s.case["steps"]
        return _outputs(s, _FLUID)
    if kind == "dem":
        s.grids[0].build(s.D.pos, 2.0 * s.r_max)
        kernels.force_dem(s.D, s.grids[0], s.r_max, s.gen.g, s.gen.dt)
        kernels.bc_dem(s.D, s.W, s.grids[1], s.rb_max, s.gen.dt)
        kernels.Kernel_step_dem(s.D, s.gen.dt)
        return {**{k: getattr(s.D, k) for k in ("force", "torque", "vel", "pos", "omega")},
                "dem_offset": s.D.contact_dem_offset_old, "bnd_offset": s.D.contact_bnd_offset_old}
    if kind == "coupling":
        solv, (gs, gb, gd, _) = s.solv, s.grids
        lo, hi = solv.dem_porosity_min, solv.dem_porosity_max
        h = s.scales[3]
        kernels.Kernel_prep_sphdem(s.P, s.B, s.D, gs, gb, gd, 2.0 * h, h, solv.support, solv.h, lo, hi)
        kernels.Kernel_interaction_dem(s.P, s.D, gs, gd, solv.mu, lo, hi, solv.dt)
        kernels.Kernel_interaction_sph(s.P, s.D, gs, gd, 2.0 * h)
        return {"P_porosity": s.P.porosity, "P_pgf": s.P.pgf, "P_acc_dem": s.P.acc_dem,
                **{"D_" + k: getattr(s.D, k) for k in ("drag", "pressure_force", "flt_s", "porosity")}}
    if kind == "kernels":
        solv, (gs, gb, _, _) = s.solv, s.grids
        kernels.Kernel_shepard_sph(s.P, s.B, gs, gb, solv.support, solv.h)
        kernels.Kernel_density_sph(s.P, s.B, gs, gb, solv.support, solv.h)
        kernels.Kernel_pres_sph(s.P, solv.rho0, solv.c0, solv.gamma)
        kernels.Kernel_force_sph(s.P, s.B, gs, gb, solv.support, solv.h, solv.mu, solv.g)
        return {k: getattr(s.P, k) for k in ("flt", "rho", "pres", "acc")}
    g, net = s.graph, s.net
    g.set_nodes(s.sets)
    g.build(check=False)
    if kind == "infer":
        return {"out": g.forward(net), "offset": g.buf["offset"][:g.n_recv + 1]}
    prepare_target(net.lib, g, s.sets, s.x_t, s.v_t, s.cfg)
    out = g.forward(net, store_pre=True)
    loss = g.loss()
    grad = g.backward(net)
    res = {"out": out.clone(), "loss": loss.clone(), "grad": grad.clone()}
    net.adam(5.0e-5)  # the end of the cosine schedule
    return res


# ---------------------------------------------------------------------------
# bytes and operations of one pass
# ---------------------------------------------------------------------------
def _counts(case):
    if case["kind"] == "ensemble":
        gens = [config_batch_member(case["first"] + i) for i in range(case["members"])]
        nf = sum(round(g.fluid_width / g.dx) * 20 * round(g.fluid_height / g.dx) for g, _, _ in gens)
        return nf, 48336 * len(gens), sum(len(p) for _, p, _ in gens)
    if case.get("scene") == "large":
        return round(case["width"] / 0.005) * 160 * 150, 2157576, case["dem"]
    nx, ny, nz = case["tx"], case["ty"], case["tz"]
    wall = (nx + 6) * (ny + 6) * (nz + 3 + 3) - nx * ny * (nz + 3)
    d = case["dem"]
    return case["fx"] * case["fy"] * case["fz"], wall, (d // 10000) * (d // 100 % 100) * (d % 100)


def work(case):
    """Each state field read once and written once; operations of the SPH pair
    sums over the support ball (~74 pairs at h = 1.3 dx; a density term is ~20
    operations, a force term ~50).  The coupling's smooth sums are counted by
    their inputs and outputs only: they need not be formed pair by pair."""
    kind = case["kind"]
    pairs = 4.0 / 3.0 * math.pi * 2.6 ** 3
    if kind == "dem":
        n = case["nx"] * case["ny"] * case["nz"]
        return {"bytes": n * (176.0 + 9 * 32 + 40), "flops": n * 8 * 150.0}
    if kind in ("infer", "train"):
        gen, pos, _ = _member(case)
        nf = round(gen.fluid_width / gen.dx) * 20 * round(gen.fluid_height / gen.dx)
        nd = gen.dem_nx * gen.dem_ny * gen.dem_nz if pos is None else len(pos)
        wall = 48336 + 14688 if case["member"] >= 0 or case["config1"] else 21000 + 6200
        edges = 30.0 * nf + 100.0 * nd
        e_flop, n_flop = 2.0 * (16 * 128 + 128 * 128), 2.0 * (16 * 128 + 128 * 128)
        rows = nf + nd + (0.2 * wall if kind == "infer" else wall)
        fwd = edges * e_flop + rows * n_flop
        byts = (nf + nd) * (60.0 + 64.0) + wall * 16.0 + edges * 8.0
        if kind == "infer":
            return {"bytes": byts, "flops": fwd}
        return {"bytes": byts + 4 * 39440 * 8.0, "flops": 3.0 * fwd + edges * e_flop}
    nf, nb, nd = _counts(case)
    steps = case.get("steps", 1)
    if kind == "coupling":
        return {"bytes": nf * 92.0 + nb * 24.0 + nd * 176.0, "flops": nf * pairs * 40.0}
    if kind == "kernels":
        return {"bytes": nf * 72.0 + nb * 36.0, "flops": nf * pairs * 80.0}
    return {"bytes": steps * (nf * 104.4 + nb * 36.0 + nd * 176.0), "flops": steps * nf * pairs * 70.0}


# ---------------------------------------------------------------------------
# the same in 64 bits, in plain torch
# ---------------------------------------------------------------------------
def _f32(x):
    return float(np.float32(x))


def _pairs(a, b, radius, ia=None, ib=None, fine=2, self_pairs=True):
    """Chunks (i, j) of the pairs with |a_i - b_j| < radius (positions in
    float32, compared in 64 bits), i ascending over the chunks."""
    if a.shape[0] == 0 or b.shape[0] == 0:
        return
    cell = radius / fine
    lo = torch.minimum(a.amin(0), b.amin(0)).double() - 2.0 * radius
    dims = ((torch.maximum(a.amax(0), b.amax(0)).double() + 2.0 * radius - lo) / cell).long() + 2
    ca, cb = ((a.double() - lo) / cell).long(), ((b.double() - lo) / cell).long()
    ncell = int(dims.prod())

    def key(c, inst):
        k = (c[:, 0] * dims[1] + c[:, 1]) * dims[2] + c[:, 2]
        return k if inst is None else k + inst.long() * ncell

    kb, order = torch.sort(key(cb, ib))
    r = range(-fine - 1, fine + 2)
    off = torch.tensor([(x, y) for x in r for y in r if max(abs(x) - 1, 0) ** 2 + max(abs(y) - 1, 0) ** 2 < fine ** 2],
                       device=a.device)
    per = max(1, int(6.0e7 / max(1.0, b.shape[0] / max(1, 1 if ib is None else int(ib.max()) + 1) * 0.02 + 400.0)))
    for i0 in range(0, a.shape[0], per):
        idx = torch.arange(i0, min(a.shape[0], i0 + per), device=a.device)
        base = key(ca[idx], None if ia is None else ia[idx])[:, None] + (off[:, 0] * dims[1] + off[:, 1]) * dims[2]
        s = torch.searchsorted(kb, (base - fine - 1).reshape(-1))
        n = torch.searchsorted(kb, (base + fine + 1).reshape(-1), right=True) - s
        rep = torch.repeat_interleave(torch.arange(n.numel(), device=a.device), n)
        j = order[s[rep] + torch.arange(rep.numel(), device=a.device) - (torch.cumsum(n, 0) - n)[rep]]
        i = idx[rep // off.shape[0]]
        keep = ((a[i].double() - b[j].double()) ** 2).sum(1) < radius * radius
        if not self_pairs:
            keep &= i != j
        yield i[keep], j[keep]


def _w(r, h):
    u = (1.0 - 0.5 * r / h).clamp_min(0.0)
    return 21.0 / (16.0 * math.pi * h ** 3) * u ** 4 * (1.0 + 2.0 * r / h)


def _dw(r, h):
    u = (1.0 - 0.5 * r / h).clamp_min(0.0)
    return -105.0 / (16.0 * math.pi * h ** 4) * (r / h) * u ** 3


class _Exact:
    """One coupled (or SPH-only) step of the state s in 64 bits."""

    def __init__(self, s, inst=None):
        self.s, self.inst = s, inst or dict(sph=None, bnd=None, dem=None, dembnd=None)
        self.h, self.rad = _f32(s.solv.h), _f32(s.solv.support)
        P, B = s.P, s.B
        d = lambda t: t.double()  # noqa: E731
        self.x, self.v, self.m, self.rho, self.flt, self.pres = (d(P.pos), d(P.vel), d(P.m), d(P.rho), d(P.flt),
                                                                 d(P.pres))
        self.xb, self.vb, self.mb, self.rhob, self.presb = d(B.pos), d(B.vel), d(B.m), d(B.rho), d(B.pres)

    def _each(self, walls=True):
        """Fluid subjects against fluid, then walls: (wall?, i, j)."""
        s, I = self.s, self.inst
        for i, j in _pairs(s.P.pos, s.P.pos, self.rad, I["sph"], I["sph"]):
            yield False, i, j
        if walls:
            for i, j in _pairs(s.P.pos, s.B.pos, self.rad, I["sph"], I["bnd"]):
                yield True, i, j

    def shepard(self):
        f = torch.zeros_like(self.rho)
        for wall, i, j in self._each():
            xj, vol = (self.xb, self.mb / self.rhob) if wall else (self.x, self.m / self.rho)
            f.index_add_(0, i, vol[j] * _w((self.x[i] - xj[j]).norm(dim=1), self.h))
        self.flt = f

    def density(self):
        r = torch.zeros_like(self.rho)
        for wall, i, j in self._each():
            xj, mj = (self.xb, self.mb) if wall else (self.x, self.m)
            r.index_add_(0, i, mj[j] * _w((self.x[i] - xj[j]).norm(dim=1), self.h))
        return r / self.flt

    def density_wall(self):
        s, I = self.s, self.inst
        r = torch.zeros_like(self.rhob)
        for nb, x, m, k in ((s.P.pos, self.x, self.m, "sph"), (s.B.pos, self.xb, self.mb, "bnd")):
            for i, j in _pairs(s.B.pos, nb, self.rad, I["bnd"], I[k]):
                r.index_add_(0, i, m[j] * _w((self.xb[i] - x[j]).norm(dim=1), self.h))
        return r

    def tait(self, rho):
        c = self.s.solv
        B = _f32(c.rho0) * _f32(c.c0) ** 2 / _f32(c.gamma)
        return B * ((rho / _f32(c.rho0)) ** _f32(c.gamma) - 1.0).clamp_min(0.0)

    def force(self):
        mu, g, h = _f32(self.s.solv.mu), _f32(self.s.solv.g), self.h
        acc, pgf = torch.zeros_like(self.x), torch.zeros_like(self.x)
        for wall, i, j in self._each():
            xj, vj, mj, rj, pj = ((self.xb, self.vb, self.mb, self.rhob, self.presb) if wall else
                                  (self.x, self.v, self.m, self.rho, self.pres))
            d = self.x[i] - xj[j]
            d2 = (d * d).sum(1)
            ok = d2 > 1.0e-12
            i, j, d, d2 = i[ok], j[ok], d[ok], d2[ok]
            r = d2.sqrt()
            gw = (_dw(r, h) / r)[:, None] * d
            sc = mj[j] * (self.pres[i] / self.rho[i] ** 2 + pj[j] / rj[j] ** 2)
            vis = mj[j] * 2.0 * mu * (d * gw).sum(1) / (self.rho[i] * rj[j]) / (d2 + 0.01 * h * h)
            acc.index_add_(0, i, vis[:, None] * (self.v[i] - vj[j]) - sc[:, None] * gw)
            pgf.index_add_(0, i, -(mj[j] / rj[j] * (pj[j] - self.pres[i]))[:, None] * gw)
        acc[:, 2] -= g
        return acc, pgf

    def too_many(self):
        """Whether the porosity's pair sums would take too long."""
        s = self.s
        if not s.D.n:
            return False
        near = self._near()
        per = 4.0 / 3.0 * math.pi * _f32(2.0 * s.scales[3]) ** 3 * _f32(s.solv.rho0) / float(s.P.m[0])
        return float(near.sum()) * min(per, s.P.n) > SEARCH_PAIRS_MAX

    def _near(self):
        s, I = self.s, self.inst
        near = torch.zeros(s.P.n, dtype=torch.bool, device=DEV)
        for i, _ in _pairs(s.P.pos, s.D.pos, 2.0 * _f32(s.scales[3]), I["sph"], I["dem"]):
            near[i] = True
        return near

    def porosity(self):
        """Fluid porosity with the fluid volumes m / rho (one coupling length h)."""
        s, I = self.s, self.inst
        h, vol = _f32(s.scales[3]), self.m / self.rho
        near = self._near().nonzero()[:, 0]
        f = torch.zeros_like(self.rho)
        sub = s.P.pos[near]
        for i, j in _pairs(sub, s.P.pos, 2.0 * h, None if I["sph"] is None else I["sph"][near], I["sph"], fine=4):
            f.index_add_(0, near[i], vol[j] * _w((self.x[near[i]] - self.x[j]).norm(dim=1), h))
        solid = torch.zeros_like(self.rho)
        xd, vd = s.D.pos.double(), s.D.volume.double()
        for i, j in _pairs(s.P.pos, s.D.pos, 2.0 * h, I["sph"], I["dem"]):
            solid.index_add_(0, i, vd[j] * _w((self.x[i] - xd[j]).norm(dim=1), h) / f[i])
        return (1.0 - solid).clamp(_f32(s.solv.dem_porosity_min), _f32(s.solv.dem_porosity_max))

    def exchange(self, pgf):
        """Drag, pressure force, volume and porosity of every sphere."""
        s, I, c = self.s, self.inst, self.s.solv
        D, h = s.D, _f32(s.scales[3])
        xd, vd, va = D.pos.double(), D.volume.double(), D.vel.double()
        f = torch.zeros(D.n, dtype=torch.float64, device=DEV)
        q = torch.zeros(D.n, 7, dtype=torch.float64, device=DEV)
        src = torch.cat([self.rho[:, None], self.v, pgf], 1)
        for j, i in _pairs(D.pos, s.P.pos, 2.0 * h, I["dem"], I["sph"], fine=4):
            w = (self.m / self.rho)[i] * _w((xd[j] - self.x[i]).norm(dim=1), h)
            f.index_add_(0, j, w)
            q.index_add_(0, j, w[:, None] * src[i])
        solid = torch.zeros_like(f)
        for i, j in _pairs(D.pos, D.pos, 2.0 * h, I["dem"], I["dem"]):
            solid.index_add_(0, i, vd[j] * _w((xd[i] - xd[j]).norm(dim=1), h))
        wet = f > 1.0e-12
        fs = torch.where(wet, f, torch.ones_like(f))
        eps = (1.0 - solid / fs).clamp(_f32(c.dem_porosity_min), _f32(c.dem_porosity_max))
        q = q / fs[:, None]
        rel = q[:, 1:4] - va
        speed, rho, mu, dia = rel.norm(dim=1), q[:, 0], _f32(c.mu), 2.0 * D.radius.double()
        re = rho * dia * speed / mu
        rr = torch.where(wet, rho, torch.ones_like(rho))
        ergun = 150.0 * (1.0 - eps) / eps * mu / dia ** 2 + 1.75 * rho * speed / dia
        cd = torch.where(re <= 1000.0, 24.0 * mu / (rr * dia) * (1.0 + 0.15 * re.clamp_min(0.0) ** 0.687),
                         0.44 * speed)
        beta = torch.where(eps <= 0.8, ergun, 0.75 * cd * rho / dia * eps ** -1.65)
        m = D.m.double()
        coef = beta * vd / m
        drag = (m * coef / (1.0 + _f32(c.dt) * coef))[:, None] * rel
        pf = (m / D.rho.double())[:, None] * q[:, 4:7]
        zero = torch.zeros_like(drag)
        hi = torch.full_like(eps, _f32(c.dem_porosity_max))
        return (torch.where(wet[:, None], drag, zero), torch.where(wet[:, None], pf, zero), f,
                torch.where(wet, eps, hi))

    def reaction(self, drag, flt_s, porosity):
        s, I = self.s, self.inst
        h = _f32(s.scales[3])
        fd = torch.zeros_like(self.x)
        xd = s.D.pos.double()
        for i, j in _pairs(s.P.pos, s.D.pos, 2.0 * h, I["sph"], I["dem"]):
            ok = flt_s[j] > 1.0e-12
            i, j = i[ok], j[ok]
            fd.index_add_(0, i, -drag[j] * (_w((self.x[i] - xd[j]).norm(dim=1), h) / flt_s[j])[:, None])
        return fd / (self.rho * porosity)[:, None]


def _contacts(D, W, g, dt, inst):
    """Gravity and contact loads of spheres without history, in 64 bits."""
    n = D.n
    x, v, w, r, m = (t.double() for t in (D.pos, D.vel, D.omega, D.radius, D.m))
    K, eta, mu = D.K.double(), D.eta.double(), D.mu.double()
    force, torque = torch.zeros_like(x), torch.zeros_like(x)
    force[:, 2] = -m * _f32(g)
    for wall in (False, True):
        nb = W if wall else D
        xn, vn, wn, rn = (t.double() for t in (nb.pos, nb.vel, nb.omega, nb.radius))
        if n == 0 or nb.n == 0:
            continue
        reach = float(r.max() + rn.max())
        for i, j in _pairs(D.pos, nb.pos, reach * 1.0001, inst["dem"], inst["dembnd" if wall else "dem"], fine=1,
                           self_pairs=wall):
            d = xn[j] - x[i]
            dist = d.norm(dim=1)
            ok = (r[i] + rn[j] - dist) > 0.0
            i, j, d, dist = i[ok], j[ok], d[ok], dist[ok]
            o = (r[i] + rn[j] - dist)[:, None]
            nrm = d / dist[:, None]
            ra, rb = (r[i][:, None] - 0.5 * o) * nrm, -(rn[j][:, None] - 0.5 * o) * nrm
            u = vn[j] + torch.linalg.cross(wn[j], rb) - v[i] - torch.linalg.cross(w[i], ra)
            un = (u * nrm).sum(1, keepdim=True) * nrm
            us = u - un
            k, e, f = K[i][:, None], eta[i][:, None], mu[i][:, None]
            fss = k * (us * _f32(dt)) + e * us
            fsf = f * k * o * us / (us.norm(dim=1, keepdim=True) + 1.0e-20)
            slide = fss.norm(dim=1, keepdim=True) >= fsf.norm(dim=1, keepdim=True)
            fs = torch.where(slide, torch.where(fss < 0.0, -1.0, 1.0) * fsf.abs(), fss)
            force.index_add_(0, i, -k * o * nrm + e * un + fs)
            torque.index_add_(0, i, torch.linalg.cross(ra, fs))
    return force, torque


def _step_dem(D, force, torque, dt):
    acc = force / D.m.double()[:, None]
    v = D.vel.double() + acc * _f32(dt)
    w = D.omega.double() + torque / D.inertia.double()[:, None] * _f32(dt)
    return {"force": force, "torque": torque, "vel": v, "pos": D.pos.double() + v * _f32(dt), "omega": w}


def exact(case, seed):
    kind = case["kind"]
    if case.get("steps", 1) != 1:
        return None
    s = prepare(case, seed)
    if kind == "dem":
        none = dict(sph=None, bnd=None, dem=None, dembnd=None)
        out = _step_dem(s.D, *_contacts(s.D, s.W, s.gen.g, s.gen.dt, none), s.gen.dt)
        return {**out, "dem_offset": None, "bnd_offset": None}
    if kind in ("infer", "train"):
        return _exact_network(s)
    inst = None
    if kind == "ensemble":
        inst = {k: g.inst for k, g in zip(("sph", "bnd", "dem", "dembnd"), s.E.grids)}
    X = _Exact(s, inst)
    if s.D.n and X.too_many():
        return None
    if kind == "kernels":
        X.shepard()
        X.rho = X.density()
        X.pres = X.tait(X.rho)
        return {"flt": X.flt, "rho": X.rho, "pres": X.pres, "acc": X.force()[0]}
    if kind == "coupling":
        por, (_, pgf) = X.porosity(), X.force()
        drag, pf, flt_s, dpor = X.exchange(pgf)
        return {"P_porosity": por, "P_pgf": pgf, "P_acc_dem": X.reaction(drag, flt_s, por), "D_drag": drag,
                "D_pressure_force": pf, "D_flt_s": flt_s, "D_porosity": dpor}
    X.shepard()  # step 0 refreshes the filter
    rho, rhob = X.density(), X.density_wall()
    X.rho, X.rhob = rho, rhob
    X.pres, X.presb = X.tait(rho), X.tait(rhob)
    acc, pgf = X.force()
    dt = _f32(s.solv.dt)
    out = {"B_rho": rhob, "B_pres": X.presb, "P_rho": rho, "P_pres": X.pres}
    if kind != "sph":
        force, torque = _contacts(s.D, s.W, s.solv.g, s.solv.dt, X.inst)
        por = X.porosity()
        drag, pf, flt_s, dpor = X.exchange(pgf)
        acc_dem = X.reaction(drag, flt_s, por)
        acc = acc + acc_dem
        dem = _step_dem(s.D, force + drag + pf, torque, s.solv.dt)
        dem.update(drag=drag, pressure_force=pf, flt_s=flt_s, porosity=dpor)
        out.update({"D_" + k: dem[k] for k in _DEM})
        out.update(P_porosity=por, P_pgf=pgf, P_acc_dem=acc_dem, dem_offset=None, bnd_offset=None)
    v = X.v + acc * dt
    out.update(P_acc=acc, P_vel=v, P_pos=X.x + v * dt)
    return out


def _exact_network(s):
    cfg, P, B, D, W = s.cfg, s.P, s.B, s.D, s.W
    d = lambda t: t.double()  # noqa: E731
    nf, nd, nb, nw = P.n, D.n, B.n, W.n
    n, nr, R = nf + nd + nb + nw, nf + nd, _f32(cfg.radius)
    pos32 = torch.cat([P.pos, D.pos, B.pos, W.pos])
    pos, vel = d(pos32), torch.zeros(n, 3, dtype=torch.float64, device=DEV)
    vel[:nr] = torch.cat([d(P.vel), d(D.vel)])
    acc = torch.cat([d(P.acc), d(D.acc)])
    X = torch.zeros(n, 16, dtype=torch.float64, device=DEV)
    X[:, 0:3] = vel / cfg.v_scale
    X[:nr, 3:6] = acc / cfg.a_scale
    X[:nf, 6], X[:nf, 7] = (d(P.rho) / cfg.rho0 - 1.0) * 100.0, d(P.porosity) - 1.0
    X[nr:nr + nb, 6] = (d(B.rho) / cfg.rho0 - 1.0) * 100.0
    X[nf:nr, 12], X[nr + nb:, 12] = d(D.radius) / R, d(W.radius) / R
    for t, (a, b) in enumerate(((0, nf), (nf, nr), (nr, nr + nb), (nr + nb, n))):
        X[a:b, 8 + t] = 1.0
    th = s.net.theta.double().requires_grad_(s.kind == "train")
    part = lambda o, r, c: th[o:o + r * c].reshape(r, c)  # noqa: E731
    E1, b1, E2, b2 = part(0, 128, 16), th[2048:2176], part(2176, 128, 128), th[18560:18688]
    N1, c1, N2, c2 = part(18688, 128, 16), th[20736:20864], part(20864, 128, 128), th[37248:37376]
    N3, c3 = part(37376, 16, 128), th[39424:39440]
    ij = [(i, j) for i, j in _pairs(pos32[:nr], pos32, R, fine=1) if i.numel()]
    i, j = torch.cat([a for a, _ in ij]), torch.cat([b for _, b in ij])
    i, j = i[i != j], j[i != j]
    dx = pos[j] - pos[i]
    e = torch.zeros(i.numel(), 16, dtype=torch.float64, device=DEV)
    e[:, 0:3], e[:, 3], e[:, 4:7] = dx / R, dx.norm(dim=1) / R, (vel[j] - vel[i]) / cfg.v_scale
    f = torch.relu(e @ E1.T + b1) @ E2.T + b2
    silu = torch.nn.functional.silu
    h0 = silu(X @ N1.T + c1)

    def gather(h):
        a = torch.zeros(nr, 128, dtype=torch.float64, device=DEV).index_add(0, i, f * h[j]) / cfg.norm
        return torch.cat([h[:nr] + a, h[nr:]])

    h2 = silu(gather(h0) @ N2.T + c2)
    out = gather(h2)[:nr] @ N3.T + c3
    if s.kind == "infer":
        return {"out": out, "offset": None}
    sx = torch.full((nr, 1), cfg.scale[0], dtype=torch.float64, device=DEV)
    sv = torch.full((nr, 1), cfg.scale[1], dtype=torch.float64, device=DEV)
    sx[nf:], sv[nf:] = cfg.scale[2], cfg.scale[3]
    m, dt = cfg.substeps, cfg.dt
    pv = vel[:nr] + m * dt * acc
    px = pos[:nr] + m * dt * vel[:nr] + 0.5 * dt * dt * m * (m + 1) * acc
    target = torch.cat([(d(s.x_t) - px) / sx, (d(s.v_t) - pv) / sv], 1)
    loss = ((out[:, :6] - target) ** 2).mean()
    loss.backward()
    return {"out": out.detach(), "loss": loss.detach().reshape(1), "grad": th.grad}
