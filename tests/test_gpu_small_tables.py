"""The one-launch stage of small tables against the two-kernel stages of large
ones: the same block is stepped alone (small) and next to an independent block
large enough that the table is not small.  FP32-flux: the same bits (the same
arithmetic on the same values, with one pressure offset).  FP64: <= 1e-14, a few
roundings of FP64, in case the compiler fuses an operation in one kernel only.

Sizes: the smallest block, boxes that divide the block and ragged ones, one-piece
and many-piece axes, the largest small table, long thin blocks, several blocks."""
import pytest
import torch

from famrdp_jax_b200.core.constants import BCType, Face
from famrdp_jax_b200.core.types import Block, BlockTopology, Config, GasModel, Metrics, SchemeChoice, State
from famrdp_jax_b200.solver.step import StepPlan
from parity_util import dev, host, random_block, rel_l2

pytestmark = pytest.mark.gpu

GAS = GasModel(gamma=1.4, R=1.0, mu0=2e-3, T0=1 / 1.4, Ts=0.27, Pr_lam=0.72)


def _plan(blocks, limiter, precision):
    """Independent blocks, periodic in i and k, farfield at the j faces."""
    F, B = Face, BCType
    topos = tuple(BlockTopology(n, {F.IMIN: (n, F.IMAX, 0), F.IMAX: (n, F.IMIN, 0), F.KMIN: (n, F.KMAX, 0),
                                    F.KMAX: (n, F.KMIN, 0)},
                                {F.IMIN: B.CUT1TO1, F.IMAX: B.CUT1TO1, F.KMIN: B.CUT1TO1, F.KMAX: B.CUT1TO1,
                                 F.JMIN: B.FARFIELD, F.JMAX: B.FARFIELD}) for n in range(len(blocks)))
    q_inf = {"q_inf": [1.0, 0.3, 0.0, 0.1, 2.0]}
    cfg = Config(gas=GAS, scheme=SchemeChoice("muscl2", "roe", 3, limiter),
                 bc_params={F.JMIN: q_inf, F.JMAX: q_inf}, topology=topos, ghost=2, nan_check=False,
                 precision=precision)
    st = State(blocks=tuple(Block(q=q, xyz=torch.zeros((3,) + tuple(q.shape[1:]), dtype=torch.float64, device="cuda"))
                            for q, _, _ in blocks),
               metrics=tuple(Metrics(jac=v, kxyz=k, vol=v) for _, k, v in blocks))
    plan = StepPlan(st, cfg)
    plan.set_p_ref(0.7 if precision == "f32" else 0.0)
    return plan


def _step(plan, qs):
    outs = [torch.full_like(q, float("nan")) for q in qs]
    plan.run(qs, outs, 1e-4)
    return outs


@pytest.mark.parametrize("precision,limiter", [("f32", "minmod"), ("f64", "minmod"), ("f64", "vanleer")])
@pytest.mark.parametrize("shapes", [[(5, 5, 5)], [(6, 7, 19)], [(8, 6, 18)], [(7, 13, 37)], [(36, 36, 36)],
                                    [(5, 5, 200)], [(300, 5, 6)], [(5, 90, 18)],
                                    [(5, 6, 7), (20, 20, 20), (9, 11, 40)]])
def test_small_tables_match_large(cuda_device, shapes, precision, limiter):
    small = [tuple(dev(x) for x in random_block(s, 40 + n)) for n, s in enumerate(shapes)]
    big = tuple(dev(x) for x in random_block((52, 48, 40), 50))
    qs = [b[0] for b in small]
    alone = _step(_plan(small, limiter, precision), qs)
    among = _step(_plan(small + [big], limiter, precision), qs + [big[0]])
    for a, b in zip(alone, among):
        assert torch.isfinite(a).all()
        if precision == "f32":
            assert torch.equal(a, b)
        else:
            assert rel_l2(host(a), host(b)) <= 1e-14


@pytest.mark.parametrize("precision", ["f32", "f64"])
@pytest.mark.parametrize("shape", [(5, 6, 9), (20, 33, 40)])
@pytest.mark.parametrize("n", [2, 8, 9, 65])
def test_tables_of_every_size_agree(cuda_device, n, shape, precision):
    """n independent blocks, all the same: tables of few, many and more blocks than a
    launch takes; every block must come out with the bits of the first."""
    one = tuple(dev(x) for x in random_block(shape, 60))
    qs = [one[0].clone() for _ in range(n)]
    outs = _step(_plan([one] * n, "minmod", precision), qs)
    ref = _step(_plan([one] * (n + 1), "minmod", precision), qs + [one[0]])
    assert torch.isfinite(ref[0]).all()
    for a in outs + ref:
        if precision == "f32":
            assert torch.equal(a, ref[0])
        else:
            assert rel_l2(host(a), host(ref[0])) <= 1e-14
