"""Volumes that are not numbers to divide by: a placeholder cell with an infinite
volume has no inviscid part, and a ghost cell that no axis differences (an edge or
corner cell of the padded block) keeps none whatever its volume is.  Blocks on both
sides of the one-launch stages' limit; the right-hand side alone and a whole step.

FP64 <= 1e-11 relative L2 of the oracle's, FP32-flux <= 1e-5, as for the other
right-hand sides; a step's change of q is dt times that.
"""
import numpy as np
import pytest
import torch

from famrdp_jax_b200.core.types import Block, BlockTopology, Config, GasModel, Metrics, SchemeChoice, State
from famrdp_jax_b200.rhs.invscd import compute_invscd_rhs
from famrdp_jax_b200.solver.step import StepPlan
from oracle.ref import NP
from parity_util import dev, host, random_block, rel_l2

pytestmark = pytest.mark.gpu

GAS = GasModel(gamma=1.4, R=1.0, mu0=2e-3, T0=1 / 1.4, Ts=0.27, Pr_lam=0.72)
SHAPES = [(9, 12, 35), (40, 44, 52)]


def _block(shape):
    q, kxyz, vol = random_block(shape, 31)
    vol[4, 5, 6] = np.inf
    vol[2, 0, shape[2] - 1] = np.inf  # differenced along i only
    vol[0, 0, 0] = np.inf
    vol[1, shape[1] - 2, 1] = np.nan
    vol[shape[0] - 1, 1, shape[2] - 2] = np.nan
    return q, kxyz, vol


@pytest.mark.parametrize("precision,bound", [("f64", 1e-11), ("f32", 1e-5)])
@pytest.mark.parametrize("shape", SHAPES)
def test_right_hand_side(cuda_device, shape, precision, bound):
    q, kxyz, vol = _block(shape)
    exp = NP.compute_invscd_rhs(q, kxyz, vol, ghost=2, gamma=1.4, limiter="minmod")
    m = Metrics(jac=dev(vol), kxyz=dev(kxyz), vol=dev(vol))
    got = host(compute_invscd_rhs(dev(q), m, ghost=2, gamma=1.4, reconstruct="muscl2", flux="roe", limiter="minmod",
                                  precision=precision))
    assert np.isfinite(exp).all() and np.isfinite(got).all()
    assert not got[:, 4, 5, 6].any() and not got[:, 0, 0, 0].any()
    for v in range(5):
        assert rel_l2(got[v], exp[v]) <= bound


@pytest.mark.parametrize("precision,bound", [("f64", 1e-11), ("f32", 1e-5)])
@pytest.mark.parametrize("shape", SHAPES)
def test_step(cuda_device, shape, precision, bound):
    q, kxyz, vol = _block(shape)
    cfg = Config(gas=GAS, scheme=SchemeChoice("muscl2", "roe", 3, "minmod"), bc_params={},
                 topology=(BlockTopology(0, {}, {}),), ghost=2, nan_check=False, precision=precision)
    exp = NP.step([q], [(kxyz, vol)], cfg, 1e-4)[0]
    st = State(blocks=(Block(q=dev(q), xyz=torch.zeros((3,) + shape, dtype=torch.float64, device="cuda")),),
               metrics=(Metrics(jac=dev(vol), kxyz=dev(kxyz), vol=dev(vol)),))
    out = torch.empty_like(st.blocks[0].q)
    StepPlan(st, cfg).run([st.blocks[0].q], [out], 1e-4)
    got = host(out)
    assert np.isfinite(exp).all() and np.isfinite(got).all()
    assert rel_l2(got - q, exp - q) <= bound
