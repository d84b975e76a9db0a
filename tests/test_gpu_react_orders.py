"""The drag reaction through the C entry with no fluid grid at all, and with one
of another particle count: point order, the same bits as in grid order."""
import ctypes as C

import numpy as np
import pytest
import torch

from helpers import scene
from warp_sph_gpt_gb300 import kernels as K
from warp_sph_gpt_gb300._lib import CtxT, check
from warp_sph_gpt_gb300.engine import context_for

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("grid", ["none", "another count"])
def test_reaction_without_a_grid_of_these_particles(grid):
    s, P, B, D, W, grids = scene(dem_nx=3, dem_ny=2, dem_origin_x=0.1, dem_origin_y=0.1, dem_spacing=0.05,
                                 dem_origin_z=0.2)
    P.vel.copy_(torch.tensor(np.random.default_rng(4).normal(0, 0.3, (P.n, 3)), dtype=torch.float32))
    P.porosity.fill_(0.9)
    K.Kernel_interaction_dem(P, D, grids[0], grids[2], s.mu, 0.05, 1.0, s.dt)
    acc0 = P.acc.clone()
    K.Kernel_interaction_sph(P, D, grids[0], grids[2], s.dem_support)
    want = P.acc_dem.clone()
    assert float(want.abs().max()) > 0
    own = context_for(P, None, D, None, (grids[0], None, grids[2], None))
    ctx = CtxT()
    C.memmove(C.byref(ctx), C.byref(own.ctx), C.sizeof(ctx))
    if grid == "none":
        ctx.grid_sph.order = ctx.grid_sph.key = ctx.grid_sph.cell_start = None
        ctx.grid_sph.n = 0
    else:
        ctx.grid_sph.n = P.n - 1
    P.acc.copy_(acc0)
    P.acc_dem.fill_(-1.0)
    check(own.lib.sphdem_interaction_sph(C.byref(ctx), s.dem_support, own.stream), "interaction_sph")
    torch.cuda.synchronize()
    assert torch.equal(P.acc_dem, want)
