"""Backward edge passes where a receiver's run of edges ends against the groups
of 8, 32 and 64 edges and the 128-edge tiles: gradients against the FP64 oracle
with the same BF16 rounding points."""
import numpy as np
import pytest
import torch

from oracle import mpnn_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("runs", [(1,), (7, 9, 8, 0, 1), (31, 33, 32, 64, 1, 63, 65), (128, 1, 127, 0, 200, 3),
                                  tuple(1 for _ in range(150)), (120,) + tuple(range(1, 24))])
def test_gradients_over_runs_of_edges(runs):
    from warp_sph_gpt_gb300.surrogate import Graph, Network, SurrogateConfig

    rng = np.random.default_rng(len(runs))
    n_recv = len(runs)
    # receiver i and its senders stand in a cluster of their own
    centre = np.stack([(np.arange(n_recv) % 13) * 0.5, (np.arange(n_recv) // 13) * 0.5, np.zeros(n_recv)], 1)
    pos = np.concatenate([centre] + [centre[i] + rng.uniform(-0.05, 0.05, (m, 3)) for i, m in enumerate(runs)])
    pos = pos.astype(np.float32)
    n = len(pos)
    vel = rng.normal(0, 0.5, size=(n, 3)).astype(np.float32)
    x = np.zeros((n, 16), np.float32)
    x[:, :10] = rng.normal(0, 1, size=(n, 10))
    x = O.bf16(x).astype(np.float32)
    cfg = SurrogateConfig(radius=0.1, dt=1e-4, rho0=1000.0, norm=8.0)
    g = Graph(cfg, "cuda")
    g._ensure(n, n_recv)
    g.n_nodes, g.n_recv = n, n_recv
    b = g.buf
    b["node_pos3"][:n] = torch.tensor(pos, device="cuda")
    b["node_pos4"][:n, :3] = torch.tensor(pos, device="cuda")
    b["node_vel4"][:n, :3] = torch.tensor(vel, device="cuda")
    b["x"][:n] = torch.tensor(x, device="cuda").to(torch.bfloat16).view(torch.int16)
    g.build()
    net = Network(cfg, "cuda", seed=5)
    net.theta[O.N3_W:O.N3_W + 768] *= 30.0
    net.pack()
    off = b["offset"][: n_recv + 1].cpu().numpy()
    own = int(np.diff(off)[0]) - runs[0]  # a receiver may be its own neighbour
    assert np.array_equal(np.diff(off), np.array(runs) + own)
    d_out = b["d_out"][:n_recv]
    d_out.zero_()
    d_out[:, :6] = torch.tensor(rng.normal(0, 1, (n_recv, 6)), dtype=torch.float32)
    g.forward(net, store_pre=True)
    grad = g.backward(net).cpu().numpy().astype(np.float64)
    assert int(g.status()) == 0
    snd = b["sender"][: off[-1]].cpu().numpy().astype(np.int64)
    rcv = b["receiver"][: off[-1]].cpu().numpy().astype(np.int64)
    pad = np.zeros((n, 1), np.float32)
    _, cache = O.forward(net.theta.cpu().numpy().astype(np.float64), x.astype(np.float64),
                         np.concatenate([pos, pad], 1), np.concatenate([vel, pad], 1), snd, rcv, n_recv,
                         1.0 / cfg.radius, 1.0 / cfg.v_scale, 1.0 / cfg.norm, quantize=True)
    gq = O.backward(cache, d_out.cpu().numpy().astype(np.float64))
    # BF16 operands (2^-9 each) through five products: the bound of the other gradient tests
    for lo, hi in ((O.E1_W, O.E1_B), (O.E1_B, O.E2_W), (O.E2_W, O.E2_B), (O.E2_B, O.N1_W), (O.N1_W, O.N1_B),
                   (O.N1_B, O.N2_W), (O.N2_W, O.N2_B), (O.N2_B, O.N3_W), (O.N3_W, O.N3_B), (O.N3_B, O.NPARAM)):
        assert np.linalg.norm(grad[lo:hi] - gq[lo:hi]) <= 3e-2 * np.linalg.norm(gq[lo:hi]) + 1e-12, (lo, hi)
