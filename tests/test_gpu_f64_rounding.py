"""Rounding errors of the FP64 path against exact values and extended precision
(NumPy's 80-bit long double).

A uniform flow through normals that are whole numbers, with a state of few bits:
every product and sum of the fluxes is exact, the dissipation is zero, and the
right-hand side must come out exact (no |n| and 1/|n| rounded into the fluxes).

The gradient of a whole right-hand side: no further off than 0.95 times what the
same expressions give in plain FP64, every operation rounded (the kernels fuse
products into sums).
"""
import numpy as np
import pytest
import torch

from dual_util import LD, DualOps, jacobian
from famrdp_jax_b200.core.types import Config, GasModel, Metrics, SchemeChoice
from famrdp_jax_b200.rhs.invscd import compute_invscd_rhs
from famrdp_jax_b200.solver.adjoint import rhs_vjp
from oracle.ref import TORCH, Ref
from parity_util import dev, host

pytestmark = [pytest.mark.gpu,
              pytest.mark.skipif(np.finfo(np.longdouble).nmant < 63, reason="long double is no wider than double")]

GAS = GasModel(gamma=1.4, R=1.0, mu0=1e-3, T0=1 / 1.4, Ts=0.27, Pr_lam=0.72)


def _rel(a, b):
    return float(np.sqrt(((a.astype(LD) - b) ** 2).sum() / (b * b).sum()))


def _state(shape, mach, amp, rng):
    def n():
        return rng.standard_normal(shape).clip(-3, 3)
    rho, p = 1 + amp * n(), (1 + amp * n()) / 1.4
    u, v, w = mach + amp * mach * n(), amp * mach * n(), amp * mach * n()
    return np.stack([rho, rho * u, rho * v, rho * w, p / 0.4 + 0.5 * rho * (u * u + v * v + w * w)])


@pytest.mark.parametrize("limiter", ["minmod", "vanleer"])
@pytest.mark.parametrize("shape", [(12, 20, 30), (40, 44, 52)])  # one and two kernels a stage
def test_uniform_flow_is_exact(cuda_device, shape, limiter):
    rng = np.random.default_rng(1)
    vel, p = np.array([0.75, -0.5625, 0.3125]), 1.25
    E = 2.0 * p + 0.5 * float(vel @ vel)  # gamma 1.5
    q = np.empty((5,) + shape)
    q[:] = np.array([1.0, *vel, E])[:, None, None, None]
    kxyz, vol = rng.integers(-32, 33, (3, 3) + shape).astype(np.float64), np.ones(shape)
    exp = np.zeros_like(q)
    for a in range(3):
        n = np.moveaxis(kxyz[a], a + 1, -1)
        n = 0.5 * (n[..., 1:-2] + n[..., 2:-1])
        un = np.einsum("m,m...->...", vel, n)
        F = np.stack([un, *[vel[m] * un + p * n[m] for m in range(3)], (E + p) * un])
        np.moveaxis(exp, a + 1, -1)[..., 2:-2] -= F[..., 1:] - F[..., :-1]
    m = Metrics(jac=dev(vol), kxyz=dev(kxyz), vol=dev(vol))
    got = host(compute_invscd_rhs(dev(q), m, ghost=2, gamma=1.5, reconstruct="muscl2", flux="roe", limiter=limiter))
    np.testing.assert_array_equal(got, exp)


def test_gradient(cuda_device):
    shape = (5, 5, 5)
    rng = np.random.default_rng(2)
    sums = np.zeros(2, dtype=LD)
    for mach in (0.2, 0.7):
        q = _state(shape, mach, 0.05, rng)
        kxyz = np.eye(3)[:, :, None, None, None] * 20.0 + 1.5 * rng.standard_normal((3, 3) + shape)
        vol = (1 / 8000.0) * (1 + 0.1 * rng.random(shape))
        cfg = Config(gas=GAS, scheme=SchemeChoice("muscl2", "roe", 3, "minmod"), bc_params={}, topology=(), ghost=2,
                     nan_check=False)
        kl, vl, ref = kxyz.astype(LD), vol.astype(LD), Ref(DualOps())
        J = jacobian(lambda x: ref.rhs_block(x, kl, vl, cfg), q)
        m = Metrics(jac=dev(vol), kxyz=dev(kxyz), vol=dev(vol))
        qt = torch.tensor(q, requires_grad=True)
        rhs = TORCH.rhs_block(qt, torch.tensor(kxyz), torch.tensor(vol), cfg)
        for _ in range(24):
            lam = rng.standard_normal(q.shape)
            exact = (J @ lam.ravel().astype(LD)).reshape(q.shape)
            plain = torch.autograd.grad((rhs * torch.tensor(lam)).sum(), qt, retain_graph=True)[0].numpy()
            got = host(rhs_vjp(dev(q), m, cfg, dev(lam)))
            sums += [_rel(plain, exact) ** 2, _rel(got, exact) ** 2]
    plain, got = np.sqrt(sums / 48)
    print(f"plain FP64 {plain:.3e}, kernels {got:.3e}")
    assert got <= 0.95 * plain
