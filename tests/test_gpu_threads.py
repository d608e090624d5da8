"""Two contexts stepped from two host threads at once (the header allows one thread
per context): small tables whose boxes need different amounts of shared memory, so
that one thread's launches must not depend on what the other's table asks for.
Every step succeeds and gives the bits it gives alone."""
import threading

import pytest
import torch

from famrdp_jax_b200 import _capi
from famrdp_jax_b200.core.types import Block, BlockTopology, Config, GasModel, Metrics, SchemeChoice, State
from famrdp_jax_b200.solver.step import StepPlan
from parity_util import dev, random_block

pytestmark = pytest.mark.gpu

GAS = GasModel(gamma=1.4, R=1.0, mu0=2e-3, T0=1 / 1.4, Ts=0.27, Pr_lam=0.72)
STEPS = 2000


def _plan(shape, precision):
    q, kxyz, vol = (dev(x) for x in random_block(shape, 70))
    cfg = Config(gas=GAS, scheme=SchemeChoice("muscl2", "roe", 3, "minmod"), bc_params={},
                 topology=(BlockTopology(0, {}, {}),), ghost=2, nan_check=False, precision=precision)
    st = State(blocks=(Block(q=q, xyz=torch.zeros((3,) + shape, dtype=torch.float64, device="cuda")),),
               metrics=(Metrics(jac=vol, kxyz=kxyz, vol=vol),))
    return StepPlan(st, cfg), q


@pytest.mark.parametrize("precision", ["f64", "f32"])
def test_two_contexts(cuda_device, precision, monkeypatch):
    # boxes of 4 x 6 x 18 and 3 x 6 x 18 cells: 129 and 104 KB in FP64, 65 and 52 in FP32
    a, qa = _plan((8, 60, 90), precision)
    with monkeypatch.context() as m:  # the second plan on a context of its own
        m.setattr(_capi, "_ctxs", {})
        b, qb = _plan((36, 36, 36), precision)
    outs, errors = [torch.empty_like(qa), torch.empty_like(qb)], []
    alone = []
    for plan, q in ((a, qa), (b, qb)):
        out = torch.empty_like(q)
        plan.run([q], [out], 1e-4)
        alone.append(out)
    torch.cuda.synchronize()

    def work(plan, q, out):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                for _ in range(STEPS):
                    plan.run([q], [out], 1e-4)
                torch.cuda.current_stream().synchronize()
        except Exception as e:  # noqa: BLE001 (reported by the test below)
            errors.append(e)

    threads = [threading.Thread(target=work, args=x) for x in ((a, qa, outs[0]), (b, qb, outs[1]))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    for out, exp in zip(outs, alone):
        assert torch.equal(out, exp)
