"""The training pass on the listed rows against the same pass on every row, and
with every buffer that a pass writes before it reads filled with NaN: rows that
take no part are neither read nor needed."""
import ctypes as C

import numpy as np
import pytest
import torch

from oracle import mpnn_oracle as O
from test_gpu_mpnn_rows import _graph

pytestmark = pytest.mark.gpu
BLOCKS = (O.E1_W, O.E1_B, O.E2_W, O.E2_B, O.N1_W, O.N1_B, O.N2_W, O.N2_B, O.N3_W, O.N3_B, O.NPARAM)


def _poison(g):
    for b, names in ((g.buf, ("z0", "h0", "agg", "h1", "z2", "h2", "h3", "out")),
                     (g.gbuf, ("g2", "d_h2", "d_h1", "d_h0", "bf_a", "bf_b", "partial"))):
        for k in names:
            if k in b:
                b[k].fill_(float("nan") if b[k].dtype == torch.float32 else 0x7fc0)  # BF16 NaN


def _unlisted(g, net):
    """Forward and backward over all rows, as without the optional lists."""
    from warp_sph_gpt_gb300 import _lib

    n, d = g._net(net), _lib.MpnnGradT()
    n.active = n.active_list = None
    d.d_out, d.grad = g.buf["d_out"].data_ptr(), net.grad.data_ptr()
    for k, t in g.gbuf.items():
        setattr(d, k, t.data_ptr())
    _lib.check(g.lib.sphdem_mpnn_forward(C.byref(n), 1, g.stream()), "forward")
    _lib.check(g.lib.sphdem_mpnn_backward(C.byref(n), C.byref(d), g.stream()), "backward")
    return net.grad


@pytest.mark.parametrize("n,n_recv", [(129, 128), (200, 1), (385, 127), (900, 640), (1400, 513)])
def test_listed_rows_are_all_that_is_needed(n, n_recv):
    from warp_sph_gpt_gb300.surrogate import Network

    g, cfg, *_ = _graph(n, n, n_recv)
    net = Network(cfg, "cuda", seed=5)
    net.theta[O.N3_W:O.N3_W + 768] *= 30.0
    net.pack()
    g.buf["d_out"][:n_recv, :6] = torch.tensor(np.random.default_rng(2).normal(0, 1, (n_recv, 6)), dtype=torch.float32)
    out = g.forward(net, store_pre=True).clone()
    g.backward(net)  # makes the workspace
    _poison(g)
    assert torch.equal(g.forward(net, store_pre=True), out)
    listed = g.backward(net).cpu().numpy().copy()
    _poison(g)
    every = _unlisted(g, net).cpu().numpy()
    assert int(g.status()) == 0 and torch.equal(g.buf["out"][:n_recv], out)
    for a, b in zip(BLOCKS, BLOCKS[1:]):
        # FP32 sums in another order, and a few BF16 steps (2^-9 of one row's share) that follow from them
        assert np.abs(listed[a:b] - every[a:b]).max() <= 2e-4 * np.abs(every[a:b]).max() + 1e-12, (a, b)
