"""The training pass on the rows that take part (receivers and the nodes that
send), and the weight-gradient kernel on a row list, at the sizes where tiles
end: against the same pass on every row and the FP64 oracle."""
import numpy as np
import pytest
import torch

from oracle import mpnn_oracle as O

pytestmark = pytest.mark.gpu


def _graph(seed, n, n_recv, radius=0.1):
    from warp_sph_gpt_gb300.surrogate import Graph, SurrogateConfig

    rng = np.random.default_rng(seed)
    pos = rng.uniform(0.0, 0.45, size=(n, 3)).astype(np.float32)
    pos[n_recv + (n - n_recv) // 2:] += 2.0  # nodes that no receiver reaches
    vel = rng.normal(0, 0.5, size=(n, 3)).astype(np.float32)
    x = np.zeros((n, 16), np.float32)
    x[:, :10] = rng.normal(0, 1, size=(n, 10))
    x = O.bf16(x).astype(np.float32)
    cfg = SurrogateConfig(radius=radius, dt=1e-4, rho0=1000.0, norm=8.0)
    g = Graph(cfg, "cuda")
    g._ensure(n, n_recv)
    g.n_nodes, g.n_recv = n, n_recv
    b = g.buf
    b["node_pos3"][:n] = torch.tensor(pos, device="cuda")
    b["node_pos4"][:n, :3] = torch.tensor(pos, device="cuda")
    b["node_vel4"][:n, :3] = torch.tensor(vel, device="cuda")
    b["x"][:n] = torch.tensor(x, device="cuda").to(torch.bfloat16).view(torch.int16)
    g.build()
    return g, cfg, np.concatenate([pos, np.zeros((n, 1), np.float32)], 1), \
        np.concatenate([vel, np.zeros((n, 1), np.float32)], 1), x.astype(np.float64)


@pytest.mark.parametrize("n,n_recv", [(129, 128), (200, 1), (385, 127), (900, 640), (1400, 513)])
def test_gradients_on_the_rows_that_take_part(n, n_recv):
    from warp_sph_gpt_gb300.surrogate import Network

    g, cfg, pos4, vel4, x = _graph(n, n, n_recv)
    net = Network(cfg, "cuda", seed=5)
    net.theta[O.N3_W:O.N3_W + 768] *= 30.0
    net.pack()
    for k in ("z0", "z2"):  # rows that take no part may hold anything
        g.buf[k].fill_(float("nan"))
    target = torch.zeros(n_recv, 16, device="cuda")
    target[:, :6] = torch.tensor(np.random.default_rng(2).normal(0, 1, (n_recv, 6)), dtype=torch.float32)
    out = g.forward(net, store_pre=True).clone()
    loss = g.loss(target).item()
    grad = g.backward(net).cpu().numpy().astype(np.float64)
    assert int(g.status()) == 0
    off = g.buf["offset"][: n_recv + 1].cpu().numpy()
    snd = g.buf["sender"][: off[-1]].cpu().numpy().astype(np.int64)
    rcv = g.buf["receiver"][: off[-1]].cpu().numpy().astype(np.int64)
    th = net.theta.cpu().numpy().astype(np.float64)
    ref, cache = O.forward(th, x, pos4, vel4, snd, rcv, n_recv, 1.0 / cfg.radius, 1.0 / cfg.v_scale, 1.0 / cfg.norm,
                           quantize=True)
    L_ref, d_out = O.loss(out.cpu().numpy().astype(np.float64), target.cpu().numpy().astype(np.float64))
    assert abs(loss - L_ref) <= 1e-5 * L_ref
    gq = O.backward(cache, d_out)
    for a, b in ((O.E1_W, O.E1_B), (O.E1_B, O.E2_W), (O.E2_W, O.E2_B), (O.E2_B, O.N1_W), (O.N1_W, O.N1_B),
                 (O.N1_B, O.N2_W), (O.N2_W, O.N2_B), (O.N2_B, O.N3_W), (O.N3_W, O.N3_B), (O.N3_B, O.NPARAM)):
        assert np.linalg.norm(grad[a:b] - gq[a:b]) <= 3e-2 * np.linalg.norm(gq[a:b]) + 1e-12, (a, b)
