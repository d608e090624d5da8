"""A block gives the same bits as a small table (one launch a stage) and in a large
one (two), in both precisions: shards of one topology, of which some are small
tables, then step bit-identically to one plan over all blocks.  The launches of each
step are counted, so that both paths are known to have run."""
import pytest
import torch

from famrdp_jax_b200 import _capi
from famrdp_jax_b200.core.constants import BCType, Face
from famrdp_jax_b200.core.types import Block, BlockTopology, Config, GasModel, Metrics, SchemeChoice, State
from famrdp_jax_b200.solver.step import StepPlan
from parity_util import dev, random_block

pytestmark = pytest.mark.gpu


def _plan(blocks, limiter, precision, law):
    """Independent blocks, periodic in i and k, walls at the j faces."""
    F, B = Face, BCType
    topos = tuple(BlockTopology(n, {F.IMIN: (n, F.IMAX, 0), F.IMAX: (n, F.IMIN, 0), F.KMIN: (n, F.KMAX, 0),
                                    F.KMAX: (n, F.KMIN, 0)},
                                {F.IMIN: B.CUT1TO1, F.IMAX: B.CUT1TO1, F.KMIN: B.CUT1TO1, F.KMAX: B.CUT1TO1,
                                 F.JMIN: B.WALL, F.JMAX: B.WALL}) for n in range(len(blocks)))
    gas = GasModel(gamma=1.4, R=1.0, mu0=2e-3, T0=1 / 1.4, Ts=0.27, Pr_lam=0.72, visc_law=law)
    cfg = Config(gas=gas, scheme=SchemeChoice("muscl2", "roe", 3, limiter), bc_params={}, topology=topos, ghost=2,
                 nan_check=False, precision=precision)
    st = State(blocks=tuple(Block(q=q, xyz=torch.zeros((3,) + tuple(q.shape[1:]), dtype=torch.float64, device="cuda"))
                            for q, _, _ in blocks),
               metrics=tuple(Metrics(jac=v, kxyz=k, vol=v) for _, k, v in blocks))
    plan = StepPlan(st, cfg)
    plan.set_p_ref(0.7 if precision == "f32" else 0.0)
    return plan


def _step(plan, qs):
    outs = [torch.full_like(q, float("nan")) for q in qs]
    n = _capi.launch_count()
    plan.run(qs, outs, 1e-4)
    return outs, _capi.launch_count() - n


@pytest.mark.parametrize("precision", ["f64", "f32"])
@pytest.mark.parametrize("limiter,law", [("minmod", "sutherland"), ("vanleer", "constant")])
@pytest.mark.parametrize("shapes", [[(5, 5, 5)], [(6, 7, 19)], [(7, 13, 37)], [(36, 36, 36)], [(5, 5, 200)],
                                    [(300, 5, 6)], [(5, 6, 7), (20, 20, 20), (9, 11, 40)]])
def test_same_bits(cuda_device, shapes, limiter, law, precision):
    small = [tuple(dev(x) for x in random_block(s, 80 + n)) for n, s in enumerate(shapes)]
    big = tuple(dev(x) for x in random_block((52, 48, 40), 90))
    qs = [b[0] for b in small]
    alone, n_alone = _step(_plan(small, limiter, precision, law), qs)
    among, n_among = _step(_plan(small + [big], limiter, precision, law), qs + [big[0]])
    assert (n_alone, n_among) == (1 + 3, 1 + 3 * 2)  # the start of the step, three stages
    for a, b in zip(alone, among):
        assert torch.isfinite(a).all()
        assert torch.equal(a, b)


@pytest.mark.parametrize("precision", ["f64", "f32"])
def test_launch_shapes_of_large_tables(cuda_device, precision):
    """Every launch shape at one and two streams on a table too large for one launch a
    stage (small ones have one shape): the same bits."""
    blocks = [tuple(dev(x) for x in random_block(s, 95 + n)) for n, s in enumerate([(40, 37, 45), (52, 48, 40)])]
    plan, qs = _plan(blocks, "minmod", precision, "sutherland"), [b[0] for b in blocks]
    ref, n = _step(plan, qs)
    assert n == 1 + 3 * 2
    for streams in (1, 2):
        plan.set_streams(streams)
        for v in range(_capi.NUM_SPLIT_VARIANTS):
            plan.set_variant(v)
            for a, b in zip(_step(plan, qs)[0], ref):
                assert torch.equal(a, b)
