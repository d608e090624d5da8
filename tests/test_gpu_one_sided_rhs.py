"""Right-hand sides with one kind of term on blocks past the one-launch stage of
small tables (two kernels, compiled for their own terms), in both flux precisions:
against the oracle, FP64 to 1e-11 as the small blocks' parity tests, FP32 fluxes to
1e-4 (the random block's fluxes cancel to about 1e-2 of their size, each rounded to
6e-8, in up to a few hundred operations).

Sizes: a ragged block just past the small tables, long thin blocks along each axis
(the shortest extents that have faces)."""
import pytest

from famrdp_jax_b200.core.types import GasModel, Metrics
from famrdp_jax_b200.rhs.invscd import compute_invscd_rhs
from famrdp_jax_b200.rhs.viscous import compute_viscous_rhs
from oracle.ref import NP
from parity_util import dev, host, random_block, rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,tol", [("f64", 1e-11), ("f32", 1e-4)])
@pytest.mark.parametrize("shape", [(35, 37, 38), (5, 6, 1700), (6, 1700, 5), (1700, 5, 6)])
def test_one_sided(cuda_device, shape, precision, tol):
    q, kxyz, vol = random_block(shape, 17)
    gas = GasModel(gamma=1.4, R=1.0, mu0=2e-3, T0=1 / 1.4, Ts=0.27, Pr_lam=0.72)
    m = Metrics(jac=dev(vol), kxyz=dev(kxyz), vol=dev(vol))
    inv = host(compute_invscd_rhs(dev(q), m, ghost=2, gamma=1.4, reconstruct="muscl2", flux="roe", limiter="vanleer",
                                  precision=precision))
    assert rel_l2(inv, NP.compute_invscd_rhs(q, kxyz, vol, ghost=2, gamma=1.4, limiter="vanleer")) <= tol
    vis = host(compute_viscous_rhs(dev(q), m, gas=gas, ghost=2, precision=precision))
    assert rel_l2(vis, NP.compute_viscous_rhs(q, kxyz, gas=gas, ghost=2)) <= tol
