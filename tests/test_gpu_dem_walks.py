"""The warp-wide walks over the spheres at the sizes where they change shape:
contact rows of no, a few, one warp's, and more contacts than the row buffer;
crowds of spheres around a few fluid particles (several tiles of 32 spheres);
the drag sums as a cluster of CTAs and as one CTA (more spheres than
clusters are used for), which give the same bits."""
import numpy as np
import pytest
import torch

from helpers import field_err, scene
from oracle.oracle import HostState
from warp_sph_gpt_gb300 import HashGrid
from warp_sph_gpt_gb300 import kernels as K
from warp_sph_gpt_gb300.struct import DEMBNDptl, DEMptl

pytestmark = pytest.mark.gpu
TOL = 1e-5


def _np(t):
    return t.detach().cpu().numpy()


def _spheres(pos, rad, rng, capacity):
    n = len(pos)
    D = DEMptl(n, "cuda", capacity_dem=capacity, capacity_bnd=max(1, capacity))
    put = lambda t, v: t.copy_(torch.tensor(np.asarray(v, np.float32)))  # noqa: E731
    put(D.pos, pos)
    put(D.vel, rng.normal(0, 0.05, (n, 3)))
    put(D.omega, rng.normal(0, 1.0, (n, 3)))
    put(D.radius, rad)
    put(D.m, 2500.0 * 4.19 * rad ** 3)
    put(D.inertia, 0.4 * 2500.0 * 4.19 * rad ** 5)
    put(D.volume, 4.19 * rad ** 3)
    D.rho.fill_(2500.0)
    D.K.fill_(2.0e4)
    D.eta.fill_(4.0)
    D.mu.fill_(0.3)
    D.h.fill_(0.08)
    return D


@pytest.mark.parametrize("m", [0, 1, 31, 32, 33, 65, 256, 257, 400])
def test_contact_rows_of_every_length(m):
    """One large sphere with m small ones on its surface, and as many wall
    spheres; three rebuilds with history."""
    rng = np.random.default_rng(m)
    u = rng.normal(0, 1, (2 * m, 3))
    u /= np.maximum(np.linalg.norm(u, axis=1, keepdims=True), 1e-9)
    big, r = 0.1, 0.004
    pos = np.concatenate([[[0.5, 0.5, 0.5]], 0.5 + u[:m] * (big + 0.9 * r)])
    D = _spheres(pos, np.concatenate([[big], np.full(m, r)]), rng, 40 * (m + 2))
    W = DEMBNDptl(max(1, m), "cuda")
    W.pos.copy_(torch.tensor(0.5 + u[m:] * (big + 0.95 * r) if m else np.full((1, 3), 9.0), dtype=torch.float32))
    W.radius.fill_(r)
    gd, gw = HashGrid(), HashGrid()
    gw.build(W.pos, 2 * big)
    for _ in range(3):
        h32, h64 = HostState(None, None, D, W), HostState(None, None, D, W)
        gd.build(D.pos, 2 * big)
        K.force_dem(D, gd, big, 9.81, 2.5e-5)
        K.bc_dem(D, W, gw, r, 2.5e-5)
        for h, p in ((h32, "f32"), (h64, "f64")):
            h.force_dem(big, 9.81, 2.5e-5, p=p)
            h.bc_dem(r, 2.5e-5, p=p)
        for kind in ("dem", "bnd"):
            ref = h32.side(kind)
            np.testing.assert_array_equal(_np(getattr(D, f"contact_{kind}_offset_old")), ref["offset"])
            np.testing.assert_array_equal(_np(getattr(D, f"contact_{kind}_id_old")), ref["id"])
            if len(ref["id"]):
                assert field_err(_np(getattr(D, f"tang_{kind}_old")), h64.side(kind)["tang"]) < TOL
        if m:
            assert int(D.contact_dem_offset_old[1]) == m and int(D.contact_bnd_offset_old[1]) == m
        assert field_err(_np(D.force), h64.dem["force"]) < TOL
        assert field_err(_np(D.torque), h64.dem["torque"]) < TOL


@pytest.mark.parametrize("n_dem", [1, 33, 300])
def test_coupling_with_crowds_of_spheres(n_dem):
    s, P, B, _, _, grids = scene()
    rng = np.random.default_rng(n_dem)
    pos = rng.uniform([0.02, 0.02, 0.02], [0.38, 0.3, 0.5], (n_dem, 3))
    D = _spheres(pos, rng.uniform(0.005, 0.02, n_dem), rng, 8)
    P.vel.copy_(torch.tensor(rng.normal(0, 0.3, (P.n, 3)), dtype=torch.float32))
    P.pres.copy_(torch.tensor(rng.uniform(0, 4e3, P.n), dtype=torch.float32))
    grids[2].build(D.pos, 0.16)
    h = HostState(P, B, D, None)
    K.Kernel_prep_sphdem(P, B, D, *grids[:3], 0.16, 0.08, s.support, s.h, 0.05, 1.0)
    K.Kernel_interaction_dem(P, D, grids[0], grids[2], s.mu, 0.05, 1.0, s.dt)
    K.Kernel_interaction_sph(P, D, grids[0], grids[2], 0.16)
    h.prep_sphdem(0.16, 0.08, s.support, s.h, 0.05, 1.0, p="f64")
    h.interaction_dem(s.mu, 0.05, 1.0, s.dt, p="f64")
    h.interaction_sph(0.16, p="f64")
    assert field_err(_np(P.porosity), h.sph["porosity"]) < TOL
    for name in ("flt_s", "porosity", "drag", "pressure_force"):
        assert field_err(_np(getattr(D, name)), h.dem[name]) < TOL, name
    assert field_err(_np(P.acc_dem), h.sph["acc_dem"]) < TOL


def test_drag_sums_of_a_cluster_and_of_one_cta():
    s, P, B, _, _, grids = scene()
    rng = np.random.default_rng(3)
    pos = rng.uniform([0.02, 0.02, 0.02], [0.38, 0.3, 0.5], (513, 3))
    pos[8:] += [0.0, 0.0, 40.0]  # beyond the reach of the first eight and of the fluid
    rad = np.full(513, 0.02)
    P.vel.copy_(torch.tensor(rng.normal(0, 0.3, (P.n, 3)), dtype=torch.float32))
    P.pgf.copy_(torch.tensor(rng.normal(0, 1.0, (P.n, 3)), dtype=torch.float32))
    got = []
    for n in (8, 513):
        D = _spheres(pos[:n], rad[:n], np.random.default_rng(1), 8)
        D.vel.zero_()
        gd = HashGrid()
        gd.build(D.pos, 0.16)
        K.Kernel_interaction_dem(P, D, grids[0], gd, s.mu, 0.05, 1.0, s.dt)
        got.append([_np(getattr(D, k))[:8] for k in ("flt_s", "porosity", "drag", "pressure_force")])
    assert np.abs(got[0][2]).max() > 0
    for a, b in zip(*got):
        np.testing.assert_array_equal(a, b)
