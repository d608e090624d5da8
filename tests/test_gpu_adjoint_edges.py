"""The RHS adjoint's face sums at the sizes where they could go wrong: the
smallest block (one face per row), rows that end inside a warp or CTA, blocks
whose last CTA is nearly empty, both limiters, both precisions.

FP64: against torch.autograd of the oracle's twin, <= 1e-10 as for the other RHS
adjoints.  FP32-flux: against the FP64 adjoint; each face's adjoint carries a few
hundred FP32 roundings of 6e-8 and minmod may switch where two slopes agree to
an FP32 rounding, which this smooth-free state makes rare: <= 1e-3.
"""
import numpy as np
import pytest
import torch

from famrdp_jax_b200.core.types import Config, GasModel, Metrics, SchemeChoice
from famrdp_jax_b200.solver.adjoint import rhs_vjp
from oracle.ref import TORCH
from parity_util import dev, host, random_block, rel_l2

pytestmark = pytest.mark.gpu

GAS = GasModel(gamma=1.4, R=1.0, mu0=2e-3, T0=1 / 1.4, Ts=0.27, Pr_lam=0.72)


def _cfg(limiter, precision):
    return Config(gas=GAS, scheme=SchemeChoice("muscl2", "roe", 3, limiter), bc_params={}, topology=(), ghost=2,
                  nan_check=False, precision=precision)


@pytest.mark.parametrize("limiter", ["minmod", "vanleer"])
@pytest.mark.parametrize("shape", [(5, 5, 5), (5, 6, 33), (9, 8, 31), (8, 17, 8), (7, 5, 130)])
def test_rhs_vjp_edges(cuda_device, shape, limiter):
    q, kxyz, vol = random_block(shape, 21)
    lam = np.random.default_rng(4).standard_normal(q.shape)
    m = Metrics(jac=dev(vol), kxyz=dev(kxyz), vol=dev(vol))
    qt = torch.tensor(q, dtype=torch.float64, requires_grad=True)
    rhs = TORCH.rhs_block(qt, torch.tensor(kxyz), torch.tensor(vol), _cfg(limiter, "f64"))
    exp = torch.autograd.grad((rhs * torch.tensor(lam)).sum(), qt)[0].numpy()
    got = host(rhs_vjp(dev(q), m, _cfg(limiter, "f64"), dev(lam)))
    assert rel_l2(got, exp) <= 1e-10
    got32 = host(rhs_vjp(dev(q), m, _cfg(limiter, "f32"), dev(lam)))
    assert rel_l2(got32, exp) <= 1e-3


@pytest.mark.parametrize("limiter", ["minmod", "vanleer"])
@pytest.mark.parametrize("mach", [0.02, 1.0, 3.0])
def test_rhs_vjp_strong_jumps(cuda_device, mach, limiter):
    """Faces with jumps of up to a factor of 20 and velocities of every sign around
    Mach ``mach``: both branches of Harten's fix on both eigenvalues, subsonic and
    supersonic (FP64, <= 1e-10: a few hundred roundings of 1e-16 of terms whose sum
    is at most 1e3 smaller than they are)."""
    shape = (6, 9, 34)
    rng = np.random.default_rng(5)
    _, kxyz, vol = random_block(shape, 22)
    rho, p = np.exp(rng.uniform(-1.5, 1.5, shape)), np.exp(rng.uniform(-1.5, 1.5, shape)) / 1.4
    u, v, w = mach * rng.standard_normal((3,) + shape)
    q = np.stack([rho, rho * u, rho * v, rho * w, p / 0.4 + 0.5 * rho * (u * u + v * v + w * w)])
    lam = rng.standard_normal(q.shape)
    m = Metrics(jac=dev(vol), kxyz=dev(kxyz), vol=dev(vol))
    qt = torch.tensor(q, dtype=torch.float64, requires_grad=True)
    rhs = TORCH.rhs_block(qt, torch.tensor(kxyz), torch.tensor(vol), _cfg(limiter, "f64"))
    exp = torch.autograd.grad((rhs * torch.tensor(lam)).sum(), qt)[0].numpy()
    assert rel_l2(host(rhs_vjp(dev(q), m, _cfg(limiter, "f64"), dev(lam))), exp) <= 1e-10
