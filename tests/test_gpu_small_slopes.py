"""The limiters of the stage kernels where the slopes of a component are too small to
multiply.  A transverse velocity v = s a, s a power of two, in a flow in which nothing
else changes along j: where s is far below the rounding of the other terms, what the
rho v equation does with v is a product with s, which is exact, or is lost beside them.
The change of rho v over a stage (without halo fill) then scales with s, down to scales
at which the product of two slopes underflows (FP32: 2^-80, FP64: 2^-560), but for
ties of roundings that v^2 breaks in a fused sum at one scale only: one rounding of a
face's terms each, relative L2 <= 1e-5 and 1e-14.  (A slope left out is 10 percent.)"""
import numpy as np
import pytest
import torch

from famrdp_jax_b200.core.types import Block, BlockTopology, Config, GasModel, Metrics, SchemeChoice, State
from famrdp_jax_b200.solver.step import StepPlan
from parity_util import dev, host, rel_l2

pytestmark = pytest.mark.gpu

GAS = GasModel(gamma=1.4, R=1.0, mu0=2e-3, T0=1 / 1.4, Ts=0.27, Pr_lam=0.72)


def _rho_v(shape, scale, precision, kernel):
    rng = np.random.default_rng(8)
    flat = np.ones(shape) * rng.standard_normal((3, shape[0], 1, shape[2]))
    rho, p, u = 1 + 0.05 * flat[0], (1 + 0.05 * flat[1]) / 1.4, 0.3 + 0.05 * flat[2]
    v = scale * rng.standard_normal(shape)
    q = dev(np.stack([rho, rho * u, rho * v, 0 * rho, p / 0.4 + 0.5 * rho * u * u]))
    vol = dev(np.full(shape, 1 / 64.0))
    st = State(blocks=(Block(q=q, xyz=torch.zeros((3,) + shape, dtype=torch.float64, device="cuda")),),
               metrics=(Metrics(jac=vol, kxyz=dev(np.eye(3)[:, :, None, None, None] * 4.0 * np.ones(shape)), vol=vol),))
    cfg = Config(gas=GAS, scheme=SchemeChoice("muscl2", "roe", 3, "minmod"), bc_params={},
                 topology=(BlockTopology(0, {}, {}),), ghost=2, nan_check=False, precision=precision)
    plan = StepPlan(st, cfg)
    if kernel == "tile":
        plan.set_kernel("tile")
    out = torch.empty_like(q)
    plan.stage([q], None, [out], 1e-3, 1)
    assert plan.check() == 0
    return (host(out)[2] / scale)[2:-2, 2:-2, 2:-2]


@pytest.mark.parametrize("shape", [(12, 14, 34), (40, 44, 52)])  # one and two kernels a stage
@pytest.mark.parametrize("precision,kernel,small,tiny,bound",
                         [("f32", "split", 50, 80, 1e-5), ("f32", "tile", 50, 80, 1e-5),
                          ("f64", "split", 90, 560, 1e-14)])
def test_rho_v_scales_with_v(cuda_device, precision, kernel, small, tiny, bound, shape):
    a, b = (_rho_v(shape, 2.0 ** -n, precision, kernel) for n in (small, tiny))
    assert rel_l2(b, a) <= bound
