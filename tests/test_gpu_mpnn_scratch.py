"""The backward pass leaves its per-CTA sums in the caller's scratch, which is
read and written by single floats: any alignment gives the same gradient."""
import numpy as np
import pytest
import torch

from test_gpu_mpnn_rows import _graph

pytestmark = pytest.mark.gpu


def test_partials_at_any_float():
    from warp_sph_gpt_gb300.surrogate import Network

    g, cfg, *_ = _graph(3, 400, 200)
    net = Network(cfg, "cuda", seed=5)
    g.buf["d_out"][:200, :6] = torch.tensor(np.random.default_rng(2).normal(0, 1, (200, 6)), dtype=torch.float32)
    g.forward(net, store_pre=True)
    want = g.backward(net).clone()
    words = g.gbuf["partial"].numel()
    g.gbuf["partial"] = torch.zeros(words + 1, dtype=torch.float32, device="cuda")[1:]
    assert g.gbuf["partial"].data_ptr() % 16 == 4
    g.forward(net, store_pre=True)
    got = g.backward(net)
    assert int(g.status()) == 0
    # the order of the atomic sums, and a BF16 step of what follows from them
    assert float((got - want).abs().max()) <= 2e-3 * float(want.abs().max())
