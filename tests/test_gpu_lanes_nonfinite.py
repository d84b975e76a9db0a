"""Non-finite positions: the several-lane loops (member slots, a small system)
give the bits of one thread per particle (walk masks), for the particles at odds
and for the others, and the step reports them."""
import numpy as np
import pytest
import torch

from helpers import scene
from warp_sph_gpt_gb300 import SPHDEM_OneStep, _lib, dem_search_scales
from warp_sph_gpt_gb300.engine import context_for
from warp_sph_gpt_gb300.simulation import check_status

pytestmark = pytest.mark.gpu
BAD = (float("nan"), float("inf"), -float("inf"), 3.0e38)


def _step(fmt):
    s, P, B, D, W, grids = scene(dem_nx=3, dem_ny=2, dem_origin_x=0.1, dem_origin_y=0.1, dem_spacing=0.05,
                                 dem_origin_z=0.2)
    scales = dem_search_scales(D, W)
    SPHDEM_OneStep(s, P, B, D, W, *grids, 0, scales)
    context_for(P, B, D, W, tuple(grids)).tuning["nbr_format"] = fmt
    for k, v in enumerate(BAD):
        P.pos[40 * k + 3, k % 3] = v
        B.pos[70 * k + 9, (k + 1) % 3] = v
    grids[1].build(B.pos, s.support)
    SPHDEM_OneStep(s, P, B, D, W, *grids, 1, scales)
    torch.cuda.synchronize()
    with pytest.raises(FloatingPointError):
        check_status(P)
    return {k: getattr(P, k).cpu().numpy() for k in ("rho", "pres", "acc", "vel", "pos")} | {"wall": B.rho.cpu().numpy()}


def test_lanes_and_one_thread_agree_on_non_finite_positions():
    lanes, one = _step(_lib.NBR_SLOTS), _step(_lib.NBR_MASKS)
    for k in lanes:
        np.testing.assert_array_equal(lanes[k], one[k], err_msg=k)
    assert np.isfinite(lanes["rho"]).mean() > 0.5
