"""Plans whose blocks have the same metrics in every cell read one cell's for all.
The same state is stepped with uniform metrics and with metrics that differ in
one value of one cell by one bit (so every cell's are read): away from that
cell's reach the results are the same bits.  The odd cell is the first, the last
and one inside; sizes on both sides of the one-launch stages' limit, two blocks
of which one is uniform."""
import pytest
import torch

from famrdp_jax_b200.core.types import Block, BlockTopology, Config, GasModel, Metrics, SchemeChoice, State
from famrdp_jax_b200.solver.step import StepPlan
from oracle.ref import NP
from parity_util import dev, host, random_block, rel_l2

pytestmark = pytest.mark.gpu

GAS = GasModel(gamma=1.4, R=1.0, mu0=2e-3, T0=1 / 1.4, Ts=0.27, Pr_lam=0.72)
REACH = 9  # three stages of two cells along each axis, and the wrap-around


def _step(qs, metrics, precision):
    topo = tuple(BlockTopology(b, {}, {}) for b in range(len(qs)))
    cfg = Config(gas=GAS, scheme=SchemeChoice("muscl2", "roe", 3, "minmod"), bc_params={}, topology=topo, ghost=2,
                 nan_check=False, precision=precision)
    xyz = torch.zeros((3, 1, 1, 1), dtype=torch.float64, device="cuda")
    st = State(blocks=tuple(Block(q=q, xyz=xyz.expand((3,) + tuple(q.shape[1:]))) for q in qs), metrics=tuple(metrics))
    outs = [torch.empty_like(q) for q in qs]
    StepPlan(st, cfg).run(qs, outs, 1e-4)
    return outs


def _uniform(shape, seed):
    _, k, _ = random_block((1, 1, 1), seed)
    kxyz = dev(k).expand((3, 3) + shape).contiguous()
    vol = torch.full(shape, 1.0 / 64.0, dtype=torch.float64, device="cuda")
    return Metrics(jac=vol, kxyz=kxyz, vol=vol)


@pytest.mark.parametrize("precision", ["f64", "f32"])
@pytest.mark.parametrize("shape", [(22, 20, 25), (40, 44, 52)])
@pytest.mark.parametrize("where", ["first", "last", "inside"])
def test_one_odd_cell(cuda_device, shape, where, precision):
    q = dev(random_block(shape, 3)[0])
    m = _uniform(shape, 5)
    odd = Metrics(jac=m.jac, kxyz=m.kxyz.clone(), vol=m.vol)
    at = {"first": (0, 0, 0), "last": tuple(n - 1 for n in shape), "inside": (0, shape[1] - 1, 1)}[where]
    v = odd.kxyz[(2, 1) + at].reshape(1)
    odd.kxyz[(2, 1) + at] = v.view(torch.int64).add(1 << 30).view(torch.float64)[0]  # one bit, kept in FP32 too
    a, b = _step([q], [m], precision)[0], _step([q], [odd], precision)[0]
    core = (slice(None),) + (slice(REACH, -REACH),) * 3
    assert torch.equal(a[core], b[core])


@pytest.mark.parametrize("precision,bound", [("f64", 1e-6), ("f32", 1e-4)])
@pytest.mark.parametrize("at", [(10, 9, 12), (2, 17, 3)])
def test_one_cell_doubled(cuda_device, at, precision, bound):
    """The change that one cell with doubled metrics makes to the step, against the
    oracle's.  The change is of the size of dt times the right-hand side there; FP64
    rounding of q is 1e-16 / 1e-4 of it a cell.  In FP32-flux the flux roundings of
    6e-8 fall on the same cells in both steps and cancel but where the change is."""
    shape = (22, 20, 25)
    q = random_block(shape, 3)[0]
    m = _uniform(shape, 5)
    odd = Metrics(jac=m.jac, kxyz=m.kxyz.clone(), vol=m.vol)
    odd.kxyz[(slice(None), slice(None)) + at] *= 2.0
    got = [host(_step([dev(q)], [x], precision)[0]) for x in (m, odd)]
    cfg = Config(gas=GAS, scheme=SchemeChoice("muscl2", "roe", 3, "minmod"), bc_params={},
                 topology=(BlockTopology(0, {}, {}),), ghost=2, nan_check=False)
    exp = [NP.step([q], [(host(x.kxyz), host(x.vol))], cfg, 1e-4)[0] for x in (m, odd)]
    assert rel_l2(got[1] - got[0], exp[1] - exp[0]) <= bound


@pytest.mark.parametrize("precision", ["f64", "f32"])
def test_uniform_next_to_general(cuda_device, precision):
    """One table with both kinds: each block as in a plan of its own."""
    shapes = [(12, 14, 20), (9, 30, 11)]
    qs, ms = [], []
    for n, s in enumerate(shapes):
        q, k, v = (dev(x) for x in random_block(s, n + 1))
        qs.append(q)
        ms.append(_uniform(s, 7) if n == 0 else Metrics(jac=v, kxyz=k, vol=v))
    both = _step(qs, ms, precision)
    if precision == "f64":  # (FP32-flux plans offset the pressure by their own blocks' mean)
        for n in range(2):
            assert torch.equal(both[n], _step([qs[n]], [ms[n]], precision)[0])
    for n in range(2):
        assert torch.isfinite(both[n]).all()
