"""Several lanes per particle (small systems) against one thread per particle
(large ones): the density, wall and force loops give the same bits.  A member
of an ensemble beyond the sizes of the several-lane loops is compared with the
same member alone, with neighbour records, without, and with records so short
that some particles overflow theirs."""
import numpy as np
import pytest
import torch

from warp_sph_gpt_gb300.batch import Case, Ensemble
from warp_sph_gpt_gb300.generate import config_batch_member

pytestmark = pytest.mark.gpu


def _stir(part, rng, lo, hi):
    """Disorder: positions off the lattice, velocities, densities off rest."""
    n = hi - lo
    part.pos[lo:hi] += torch.tensor(rng.uniform(-4e-4, 4e-4, (n, 3)), dtype=torch.float32, device="cuda")
    part.vel[lo:hi] = torch.tensor(rng.normal(0.0, 0.2, (n, 3)), dtype=torch.float32, device="cuda")
    part.rho[lo:hi] *= torch.tensor(rng.uniform(0.998, 1.002, n), dtype=torch.float32, device="cuda")


@pytest.mark.parametrize("nbr_cap", [-1, 0, 60])
def test_lanes_give_the_bits_of_one_thread(nbr_cap):
    ids = list(range(14))
    members = [config_batch_member(i) for i in ids]
    ens = Ensemble(members)
    assert ens.P.n > 128 * 1024 and ens.B.n > 256 * 1024
    ens.tune({"nbr_cap": nbr_cap})
    o = ens.offsets["sph"]
    for k in ids:
        _stir(ens.P, np.random.default_rng(k), int(o[k]), int(o[k + 1]))
    ens.run(0, 3)
    for k in (0, 5, 13):
        alone = Case(*members[k])
        assert alone.P.n < 64 * 1024
        alone.tune({"nbr_cap": nbr_cap})
        _stir(alone.P, np.random.default_rng(k), 0, alone.P.n)
        alone.run(0, 3)
        for field in ("rho", "pres", "flt", "acc", "pgf", "vel", "pos"):
            np.testing.assert_array_equal(ens.member(k, "sph", field).cpu().numpy(),
                                          getattr(alone.P, field).cpu().numpy(), err_msg=f"member {k} {field}")
        np.testing.assert_array_equal(ens.member(k, "bnd", "rho").cpu().numpy(), alone.B.rho.cpu().numpy())


@pytest.mark.parametrize("n", [1, 3, 31, 33, 257])
def test_sparse_and_scattered_particles(n):
    """Few particles, most in columns of their own, some outside the cell box
    and one pair closer than the force's minimum distance."""
    from warp_sph_gpt_gb300 import HashGrid, kernels
    from warp_sph_gpt_gb300.struct import BNDptl, SPHptl

    rng = np.random.default_rng(n)
    P, B = SPHptl(n, "cuda"), BNDptl(5, "cuda")
    for part in (P, B):
        part.pos.copy_(torch.tensor(rng.uniform(0.0, 0.6, (part.n, 3)), dtype=torch.float32))
        part.m.fill_(0.008)
        part.rho.fill_(1000.0)
    grids = [HashGrid(), HashGrid()]
    for g, part in zip(grids, (P, B)):
        g.build(part.pos, 0.2)
    kernels.Kernel_shepard_sph(P, B, *grids, 0.2, 0.1)  # fixes the cell box
    P.pos[n // 2] = torch.tensor([3.0, -2.0, 9.0])
    if n > 3:
        P.pos[1] = P.pos[0] + torch.tensor([5e-7, 0.0, 0.0], device="cuda")
    kernels.Kernel_shepard_sph(P, B, *grids, 0.2, 0.1)
    kernels.Kernel_density_sph(P, B, *grids, 0.2, 0.1)
    kernels.Kernel_force_sph(P, B, *grids, 0.2, 0.1, 0.05, 9.81)
    x, xb = P.pos.double().cpu().numpy(), B.pos.double().cpu().numpy()
    d = np.linalg.norm(x[:, None] - np.concatenate([x, xb])[None], axis=-1)
    u = np.maximum(1.0 - 0.5 * d / 0.1, 0.0)
    w = 21.0 / (16.0 * np.pi * 0.1 ** 3) * u ** 4 * (1.0 + 2.0 * d / 0.1)
    flt = (0.008 / 1000.0 * w).sum(1)
    np.testing.assert_allclose(P.flt.cpu().numpy(), flt, rtol=2e-6, atol=1e-9)
    np.testing.assert_allclose(P.rho.cpu().numpy(), 1000.0, rtol=4e-6)
    assert torch.isfinite(P.acc).all()


@pytest.mark.parametrize("n", [5000, 66000])
@pytest.mark.parametrize("support", [0.03, 0.05])
def test_sums_with_a_support_that_is_not_the_kernels(n, support):
    """A support beyond 2 h, whose outer members weigh nothing, and one below,
    which cuts the kernel off: several lanes (5,000) and one thread (66,000)."""
    from scipy.spatial import cKDTree

    from warp_sph_gpt_gb300 import HashGrid, kernels
    from warp_sph_gpt_gb300.struct import BNDptl, SPHptl

    h = 0.02
    rng = np.random.default_rng(n)
    P, B = SPHptl(n, "cuda"), BNDptl(7, "cuda")
    side = (n / 60.0 * (4.0 / 3.0) * np.pi * (2.0 * h) ** 3) ** (1.0 / 3.0)  # ~60 neighbours
    for part in (P, B):
        part.pos.copy_(torch.tensor(rng.uniform(0.0, side, (part.n, 3)), dtype=torch.float32))
        part.m.fill_(0.008)
        part.rho.fill_(1000.0)
    grids = [HashGrid(), HashGrid()]
    for g, part in zip(grids, (P, B)):
        g.build(part.pos, support)
    kernels.Kernel_shepard_sph(P, B, *grids, support, h)
    x = np.concatenate([P.pos.double().cpu().numpy(), B.pos.double().cpu().numpy()])
    some = rng.choice(n, 300, replace=False)
    want = np.empty(300)
    for i, j in enumerate(cKDTree(x).query_ball_point(x[some], support)):
        q = np.linalg.norm(x[j] - x[some[i]], axis=1) / h
        want[i] = (0.008 / 1000.0 * 21.0 / (16.0 * np.pi * h ** 3) * np.maximum(1 - 0.5 * q, 0) ** 4 * (1 + 2 * q)).sum()
    # ~120 additions and a dozen roundings a term of 2^-24, twice that for the FP32 positions
    np.testing.assert_allclose(P.flt.cpu().numpy()[some], want, rtol=2e-5)
