"""Uniform blocks (every cell the same metrics: one cell's are read for all) next to
general ones, and blocks that differ from uniform in one value of one cell anywhere.

The pressure offset of the FP32-flux plans is set to one value, so that a block has
the same bits whatever its neighbours in the table are."""
import numpy as np
import pytest
import torch

from famrdp_jax_b200.core.types import Block, BlockTopology, Config, GasModel, Metrics, SchemeChoice, State
from famrdp_jax_b200.solver.step import StepPlan
from parity_util import dev, random_block

pytestmark = pytest.mark.gpu

GAS = GasModel(gamma=1.4, R=1.0, mu0=2e-3, T0=1 / 1.4, Ts=0.27, Pr_lam=0.72)


def _step(qs, metrics, precision):
    topo = tuple(BlockTopology(b, {}, {}) for b in range(len(qs)))
    cfg = Config(gas=GAS, scheme=SchemeChoice("muscl2", "roe", 3, "minmod"), bc_params={}, topology=topo, ghost=2,
                 nan_check=False, precision=precision)
    xyz = torch.zeros((3, 1, 1, 1), dtype=torch.float64, device="cuda")
    st = State(blocks=tuple(Block(q=q, xyz=xyz.expand((3,) + tuple(q.shape[1:]))) for q in qs), metrics=tuple(metrics))
    outs = [torch.empty_like(q) for q in qs]
    plan = StepPlan(st, cfg)
    plan.set_p_ref(0.7 if precision == "f32" else 0.0)
    plan.run(qs, outs, 1e-3)
    return outs


def _uniform(shape, seed):
    _, k, _ = random_block((1, 1, 1), seed)
    vol = torch.full(shape, 1.0 / 64.0, dtype=torch.float64, device="cuda")
    return Metrics(jac=vol, kxyz=dev(k).expand((3, 3) + shape).contiguous(), vol=vol)


@pytest.mark.parametrize("precision", ["f64", "f32"])
@pytest.mark.parametrize("shapes", [[(12, 14, 20), (9, 30, 11), (8, 9, 10)], [(40, 44, 52), (12, 50, 31), (33, 20, 41)]])
@pytest.mark.parametrize("kinds", ["ugg", "gug", "uug", "guu"])
def test_mixed_table(cuda_device, kinds, shapes, precision):
    """One table of uniform (u) and general (g) blocks: each as in a plan of its own."""
    qs, ms = [], []
    for n, (kind, s) in enumerate(zip(kinds, shapes)):
        q, k, v = (dev(x) for x in random_block(s, n + 1))
        qs.append(q)
        ms.append(_uniform(s, 7 + n) if kind == "u" else Metrics(jac=v, kxyz=k, vol=v))
    for a, q, m in zip(_step(qs, ms, precision), qs, ms):
        assert torch.isfinite(a).all()
        assert torch.equal(a, _step([q], [m], precision)[0])


@pytest.mark.parametrize("precision", ["f64", "f32"])
@pytest.mark.parametrize("shape", [(22, 24, 25), (40, 44, 52)])
def test_one_odd_cell_anywhere(cuda_device, shape, precision):
    """One value doubled in one interior cell, alone and with a second odd cell in the
    first corner, which makes the block general beyond doubt: the same bits beyond
    that corner's reach (three stages of two cells and the wrap-around), the odd cell
    itself among them, and not those of the uniform block."""
    rng = np.random.default_rng(6)
    q, m = dev(random_block(shape, 3)[0]), _uniform(shape, 5)
    plain = _step([q], [m], precision)[0]
    core = (slice(None),) + (slice(9, -9),) * 3
    for n in range(18):
        at = tuple(int(rng.integers(10, s - 10)) for s in shape)
        odd = m.kxyz.clone()
        odd[(n % 9 // 3, n % 3) + at] *= 2.0
        both = odd.clone()
        both[:, :, 0, 0, 0] *= 2.0
        a, b = (_step([q], [Metrics(jac=m.jac, kxyz=k, vol=m.vol)], precision)[0] for k in (odd, both))
        assert torch.equal(a[core], b[core])
        assert not torch.equal(a[core], plain[core])
