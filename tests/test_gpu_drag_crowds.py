"""Drag and solid fraction of crowds of wet spheres, on both sides of the count
up to which a cluster of CTAs shares a sphere, with few and with many columns in
a sphere's window (their candidates are dealt out to the warps 32 at a time)."""
import numpy as np
import pytest
import torch

from helpers import field_err, scene
from oracle.oracle import HostState
from warp_sph_gpt_gb300 import HashGrid
from warp_sph_gpt_gb300 import kernels as K
from warp_sph_gpt_gb300.struct import DEMptl

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [512, 513])
@pytest.mark.parametrize("cell", [0.16, 0.021])
def test_crowds_of_wet_spheres(n, cell):
    s, P, B, _, _, grids = scene()
    rng = np.random.default_rng(n)
    rad = rng.uniform(0.003, 0.006, n)
    D = DEMptl(n, "cuda", capacity_dem=8, capacity_bnd=8)
    put = lambda t, v: t.copy_(torch.tensor(np.asarray(v, np.float32)))  # noqa: E731
    put(D.pos, rng.uniform([0.0, 0.0, 0.0], [0.4, 0.3, 0.45], (n, 3)))
    put(D.vel, rng.normal(0, 0.1, (n, 3)))
    put(D.radius, rad)
    put(D.m, 2500.0 * 4.19 * rad ** 3)
    put(D.volume, 4.19 * rad ** 3)
    D.rho.fill_(2500.0)
    D.h.fill_(0.08)
    put(P.vel, rng.normal(0, 0.3, (P.n, 3)))
    put(P.pgf, rng.normal(0, 1.0, (P.n, 3)))
    gd = HashGrid()
    gd.build(D.pos, cell)
    h = HostState(P, B, D, None)
    K.Kernel_interaction_dem(P, D, grids[0], gd, s.mu, 0.05, 1.0, s.dt)
    h.interaction_dem(s.mu, 0.05, 1.0, s.dt, p="f64")
    for name in ("flt_s", "porosity", "drag", "pressure_force"):
        assert field_err(getattr(D, name).cpu().numpy(), h.dem[name]) < 1e-5, name
