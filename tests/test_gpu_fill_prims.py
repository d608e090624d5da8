"""The step's start: the copy, halo fill and boundary faces that also write the
stage-1 primitives.  A step into other arrays takes that path; the same step in
place copies, fills and computes the primitives in separate kernels.  Both must
give the same bits, at cell counts around the CTA sizes (one and four cells per
thread), with every boundary type and a mapped interface."""
import pytest
import torch

from famrdp_jax_b200.core.constants import BCType, Face, mapped_orientation
from famrdp_jax_b200.core.types import Block, BlockTopology, Config, GasModel, Metrics, SchemeChoice, State
from famrdp_jax_b200.solver.step import StepPlan
from parity_util import dev, random_block

pytestmark = pytest.mark.gpu

GAS = GasModel(gamma=1.4, R=1.0, mu0=2e-3, T0=1 / 1.4, Ts=0.27, Pr_lam=0.72)


def _topology():
    """Two blocks: block 0 periodic in i with an isothermal wall and a symmetry
    plane along j and a farfield face along k, joined at its k-max face to block
    1's k-max face in a mapped orientation; block 1's other faces adiabatic
    walls, periodic in j."""
    F, B = Face, BCType
    t0 = BlockTopology(0, {F.IMIN: (0, F.IMAX, 0), F.IMAX: (0, F.IMIN, 0),
                           F.KMAX: (1, F.KMAX, mapped_orientation(reverse_a=True))},
                       {F.IMIN: B.CUT1TO1, F.IMAX: B.CUT1TO1, F.JMIN: B.WALL, F.JMAX: B.SYMMETRY,
                        F.KMIN: B.FARFIELD, F.KMAX: B.CUT1TO1})
    t1 = BlockTopology(1, {F.KMAX: (0, F.KMAX, mapped_orientation(reverse_a=True)), F.JMIN: (1, F.JMAX, 0),
                           F.JMAX: (1, F.JMIN, 0)},
                       {F.KMAX: B.CUT1TO1, F.JMIN: B.CUT1TO1, F.JMAX: B.CUT1TO1, F.IMIN: B.SYMMETRY,
                        F.IMAX: B.FARFIELD, F.KMIN: B.WALL})
    prm = {F.JMIN: {"wall_type": "isothermal", "T_wall": 0.9}, F.KMIN: {"q_inf": [1.0, 0.3, 0.0, 0.1, 2.0]},
           F.IMAX: {"q_inf": [1.1, 0.2, 0.1, 0.0, 2.1]}}
    return (t0, t1), prm


@pytest.mark.parametrize("precision", ["f64", "f32"])
@pytest.mark.parametrize("nij,nk0,nk1", [((7, 9), 5, 8), ((16, 32), 16, 5), ((101, 83), 77, 6), ((64, 128), 80, 128)])
def test_fill_with_primitives_matches_separate_kernels(cuda_device, nij, nk0, nk1, precision):
    topo, prm = _topology()
    cfg = Config(gas=GAS, scheme=SchemeChoice("muscl2", "roe", 3, "minmod"), bc_params=prm, topology=topo, ghost=2,
                 nan_check=False, precision=precision)
    blocks, metrics = [], []
    for b, nk in enumerate((nk0, nk1)):
        q, kxyz, vol = random_block(nij + (nk,), b + 1)
        blocks.append(Block(q=dev(q), xyz=torch.zeros((3,) + q.shape[1:], dtype=torch.float64, device="cuda")))
        metrics.append(Metrics(jac=dev(vol), kxyz=dev(kxyz), vol=dev(vol)))
    state = State(blocks=tuple(blocks), metrics=tuple(metrics))
    plan = StepPlan(state, cfg)
    qs = [b.q for b in blocks]
    keep = [q.clone() for q in qs]
    outs = [torch.full_like(q, float("nan")) for q in qs]
    plan.run(qs, outs, 1e-5)
    same = [q.clone() for q in qs]
    plan.run(same, same, 1e-5)
    for q, k, o, s in zip(qs, keep, outs, same):
        assert torch.equal(q, k)  # the input is untouched
        assert torch.equal(o, s)
        assert torch.isfinite(o).all()


@pytest.mark.parametrize("precision", ["f64", "f32"])
@pytest.mark.parametrize("shape", [(5, 5, 5), (6, 5, 9), (9, 12, 33)])
def test_boundary_faces_alone(cuda_device, shape, precision):
    """No interface at all: every ghost cell comes from boundary faces, edges and
    corners through up to three of them, thin blocks through both faces of an
    axis."""
    F, B = Face, BCType
    topo = (BlockTopology(0, {}, {F.IMIN: B.WALL, F.IMAX: B.SYMMETRY, F.JMIN: B.SYMMETRY, F.JMAX: B.WALL,
                                  F.KMIN: B.WALL, F.KMAX: B.FARFIELD}),)
    prm = {F.JMAX: {"wall_type": "isothermal", "T_wall": 0.8}, F.KMAX: {"q_inf": [1.0, 0.3, 0.0, 0.1, 2.0]}}
    cfg = Config(gas=GAS, scheme=SchemeChoice("muscl2", "roe", 3, "minmod"), bc_params=prm, topology=topo, ghost=2,
                 nan_check=False, precision=precision)
    q, kxyz, vol = (dev(x) for x in random_block(shape, 9))
    state = State(blocks=(Block(q=q, xyz=torch.zeros((3,) + shape, dtype=torch.float64, device="cuda")),),
                  metrics=(Metrics(jac=vol, kxyz=kxyz, vol=vol),))
    plan = StepPlan(state, cfg)
    out = torch.full_like(q, float("nan"))
    plan.run([q], [out], 1e-5)
    same = q.clone()
    plan.run([same], [same], 1e-5)
    assert torch.equal(out, same)
