"""A query radius below the spheres' reach 2 h_b: which spheres a particle sees
is decided by the cells of its own window, not by the particles whose warp it
shares.  The reaction against the FP64 sum over those spheres, and the particles
that the porosity pass takes for dry."""
import numpy as np
import pytest
import torch

from helpers import field_err, scene
from warp_sph_gpt_gb300 import kernels as K
from warp_sph_gpt_gb300.struct import DEMptl

pytestmark = pytest.mark.gpu


def _w(r, h):
    q = r / h
    return np.where(q < 2.0, 21.0 / (16.0 * np.pi * h ** 3) * np.maximum(1.0 - 0.5 * q, 0.0) ** 4 * (1.0 + 2.0 * q), 0.0)


def _cells(x, geometry):
    lo, dim, _, inv = geometry
    c = np.floor(x.astype(np.float32) * np.float32(inv)).astype(np.int64) - np.array(lo)
    return np.clip(c, 0, np.array(dim) - 1)


def _seen(x, xs, support, geometry):
    """[particle, sphere]: the sphere's cell overlaps the particle's window."""
    rq = np.float32(np.float32(support) * np.float32(1.001) + np.float32(1e-6))
    a, b, c = _cells(x - rq, geometry), _cells(x + rq, geometry), _cells(xs, geometry)
    return ((c[None] >= a[:, None]) & (c[None] <= b[:, None])).all(-1)


@pytest.mark.parametrize("support", [0.02, 0.06, 0.16])
def test_spheres_of_a_particles_own_window(support):
    s, P, B, _, _, grids = scene()
    rng = np.random.default_rng(11)
    n, h = 40, 0.08
    D = DEMptl(n, "cuda", capacity_dem=8, capacity_bnd=8)
    D.pos.copy_(torch.tensor(rng.uniform([0.0, 0.0, 0.0], [0.5, 0.3, 0.5], (n, 3)), dtype=torch.float32))
    D.h.fill_(h)
    D.volume.fill_(3e-5)
    grids[2].build(D.pos, 0.06)
    P.porosity.fill_(1.0)
    K.Kernel_prep_sphdem(P, B, D, *grids[:3], support, h, s.support, s.h, 0.05, 1.0)
    porosity = P.porosity.cpu().numpy()
    D.drag.copy_(torch.tensor(rng.normal(0, 1, (n, 3)), dtype=torch.float32))
    D.flt_s.fill_(1.5)
    K.Kernel_interaction_sph(P, D, grids[0], grids[2], support)
    x, xs = P.pos.cpu().numpy(), D.pos.cpu().numpy()
    d = np.linalg.norm(x[:, None].astype(float) - xs[None].astype(float), axis=-1)
    reach = d < 2.0 * h
    seen = reach & _seen(x, xs, support, grids[2].geometry)
    if support < 0.1:
        assert (seen.sum(1) < reach.sum(1)).any()
    w = np.where(seen, _w(d, h), 0.0)
    den = (P.rho.double() * P.porosity.double()).cpu().numpy()
    want = -(w[:, :, None] * D.drag.double().cpu().numpy()[None] / 1.5).sum(1) / den[:, None]
    assert field_err(P.acc_dem.cpu().numpy(), want) < 1e-5
    # the porosity pass's normaliser is for a query radius of 2 h; its list of
    # particles with spheres, and so where the porosity is not 1, for any
    none = ~seen.any(1)
    assert none.any() and (porosity[none] == 1.0).all()
    assert (porosity[(w * 3e-5).sum(1) > 1e-3] < 1.0).all()
