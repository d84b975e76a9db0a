"""The grid build against a stable NumPy sort by cell, at the sizes where its
paths meet: one CTA or several kernels, cells of a few points (ranked), cells
beyond the ranked length (sorted by the whole CTA, in shared memory or in
place), cells that straddle a CTA's window, cell counts that end inside a scan
tile or span."""
import numpy as np
import pytest
import torch

from warp_sph_gpt_gb300 import HashGrid
from warp_sph_gpt_gb300.engine import context_for
from warp_sph_gpt_gb300.struct import SPHptl

pytestmark = pytest.mark.gpu


def _points(n, clump, box, rng):
    """n points in the box, `clump` of them inside one tenth of a cell."""
    pos = rng.uniform(0.0, 1.0, (n, 3)) * box
    if clump:
        pos[rng.permutation(n)[:clump]] = np.array(box) * 0.5 + rng.uniform(0.01, 0.1, (clump, 3)) * 0.1
    return pos.astype(np.float32)


@pytest.mark.parametrize("n,clump,box", [
    (1, 0, (1, 1, 1)), (255, 0, (1, 1, 1)), (4096, 0, (2, 1, 1)), (4096, 64, (1, 1, 1)), (4095, 65, (1, 1, 1)),
    (3000, 2900, (1, 1, 1)), (4097, 0, (1, 1, 1)), (5000, 769, (1, 1, 1)), (5000, 1100, (1, 1, 1)),
    (9001, 4096, (1, 1, 1)), (9001, 4097, (2, 1, 1)), (20000, 12345, (3, 1, 1)), (70001, 300, (9, 3, 2)),
    (33333, 0, (50, 25, 13)),
])
def test_cells_are_sorted_stably(n, clump, box):
    rng = np.random.default_rng(n + clump)
    pos = _points(n, clump, box, rng)
    P = SPHptl(n, "cuda")
    P.pos.copy_(torch.tensor(pos))
    P.m.copy_(torch.tensor(rng.uniform(0.5, 1.5, n).astype(np.float32)))
    P.rho.fill_(1000.0)
    g = HashGrid()
    g.build(P.pos, 0.1)
    ctx = context_for(P, None, None, None, (g, None, None, None))
    ctx.prepare()
    torch.cuda.synchronize()
    lo, dim, cell, inv = g.geometry
    c = np.floor(pos * np.float32(inv)).astype(np.int64) - np.array(lo)
    key = (c[:, 0] * dim[1] + c[:, 1]) * dim[2] + c[:, 2]
    np.testing.assert_array_equal(g.cell_keys().cpu().numpy(), key)
    order = np.argsort(key, kind="stable")
    np.testing.assert_array_equal(g.sorted_order().cpu().numpy(), order)
    start = np.searchsorted(key[order], np.arange(dim[0] * dim[1] * dim[2] + 1))
    np.testing.assert_array_equal(g.buffers["cell_start"].cpu().numpy(), start)
    posm = ctx.work["f_posm"].cpu().numpy()
    np.testing.assert_array_equal(posm[:, :3], pos[order])
    np.testing.assert_array_equal(posm[:, 3], P.m.cpu().numpy()[order])
