"""The reverse of the limiters where the slopes are too small to multiply.

With a transverse velocity v = s a, s tiny, the rho v equation is homogeneous of
degree one in v (v enters the other terms relative to the speed of sound), so its
gradient with respect to rho v does not depend on s.  s is a power of two: every
product with v is scaled exactly, and the gradients at two scales differ by the
terms of order s and by the roundings these flip: <= 1e-5 in FP32 (a few of 6e-8),
<= 1e-14 in FP64.  At the smaller scale the product of two slopes underflows.
"""
import numpy as np
import pytest

from famrdp_jax_b200.core.types import Config, GasModel, Metrics, SchemeChoice
from famrdp_jax_b200.solver.adjoint import rhs_vjp
from parity_util import dev, host, rel_l2

pytestmark = pytest.mark.gpu

GAS = GasModel(gamma=1.4, R=1.0, mu0=2e-3, T0=1 / 1.4, Ts=0.27, Pr_lam=0.72)


def _gradient(scale, precision):
    shape = (9, 10, 33)
    rng = np.random.default_rng(8)
    rho = 1 + 0.05 * rng.standard_normal(shape)
    p = (1 + 0.05 * rng.standard_normal(shape)) / 1.4
    u = 0.3 + 0.05 * rng.standard_normal(shape)
    v = scale * rng.standard_normal(shape)
    q = np.stack([rho, rho * u, rho * v, 0 * rho, p / 0.4 + 0.5 * rho * u * u])
    lam = np.zeros_like(q)
    lam[2] = rng.standard_normal(shape)
    kxyz = np.eye(3)[:, :, None, None, None] * 4.0 * np.ones(shape)
    vol = np.full(shape, 1 / 64.0)
    cfg = Config(gas=GAS, scheme=SchemeChoice("muscl2", "roe", 3, "minmod"), bc_params={}, topology=(), ghost=2,
                 nan_check=False, precision=precision)
    m = Metrics(jac=dev(vol), kxyz=dev(kxyz), vol=dev(vol))
    return host(rhs_vjp(dev(q), m, cfg, dev(lam)))[2]


@pytest.mark.parametrize("precision,small,tiny,bound", [("f32", 40, 90, 1e-5), ("f64", 60, 560, 1e-14)])
def test_gradient_does_not_depend_on_the_scale(cuda_device, precision, small, tiny, bound):
    exp, got = _gradient(2.0 ** -small, precision), _gradient(2.0 ** -tiny, precision)
    assert np.linalg.norm(exp) > 1.0
    assert rel_l2(got, exp) <= bound
