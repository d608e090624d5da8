"""The FP64 face flux (MUSCL + Roe with grouped sums) where its regroupings and
selections matter: strong jumps and supersonic faces in every direction, both
limiters, Harten's branch on both eigenvalues, cells whose face normals vanish,
and the reach of a non-finite cell.

Tolerance: relative L2 <= 1e-11 of the inviscid right-hand side, as for the other
RHS fields (an ulp of a face flux is |F| / |dF| ulp of the difference; the
regrouped sums differ from the plain ones by a few ulp of the face's terms).
"""
import numpy as np
import pytest

from famrdp_jax_b200.core.types import Metrics
from famrdp_jax_b200.rhs.invscd import compute_invscd_rhs
from oracle.ref import NP
from parity_util import dev, host, random_block, rel_l2

pytestmark = pytest.mark.gpu


def _strong_block(shape, seed, mach):
    """Cell-to-cell jumps of up to a factor of 20 in density and pressure, and
    velocities of every sign around Mach ``mach``."""
    rng = np.random.default_rng(seed)
    _, kxyz, vol = random_block(shape, seed)
    rho = np.exp(rng.uniform(-1.5, 1.5, shape))
    p = np.exp(rng.uniform(-1.5, 1.5, shape)) / 1.4
    u, v, w = mach * rng.standard_normal((3,) + shape)
    return np.stack([rho, rho * u, rho * v, rho * w, p / 0.4 + 0.5 * rho * (u * u + v * v + w * w)]), kxyz, vol


def _rhs(q, kxyz, vol, limiter):
    m = Metrics(jac=dev(vol), kxyz=dev(kxyz), vol=dev(vol))
    return host(compute_invscd_rhs(dev(q), m, ghost=2, gamma=1.4, reconstruct="muscl2", flux="roe", limiter=limiter))


@pytest.mark.parametrize("limiter", ["minmod", "vanleer"])
@pytest.mark.parametrize("shape,mach", [((9, 12, 35), 0.02), ((5, 5, 5), 1.0), ((6, 31, 64), 3.0)])
def test_strong_jumps(cuda_device, shape, mach, limiter):
    q, kxyz, vol = _strong_block(shape, 3, mach)
    exp = NP.compute_invscd_rhs(q, kxyz, vol, ghost=2, gamma=1.4, limiter=limiter)
    got = _rhs(q, kxyz, vol, limiter)
    for v in range(5):
        assert rel_l2(got[v], exp[v]) <= 1e-11


def test_vanishing_normals(cuda_device):
    """Faces whose averaged normal is zero (degenerate metrics) carry no flux."""
    q, kxyz, vol = _strong_block((9, 10, 33), 5, 0.5)
    kxyz[0, :, 3:6] = 0.0
    kxyz[2, :, :, :, 10:20] = 0.0
    exp = NP.compute_invscd_rhs(q, kxyz, vol, ghost=2, gamma=1.4, limiter="minmod")
    got = _rhs(q, kxyz, vol, "minmod")
    assert np.isfinite(got).all()
    for v in range(5):
        assert rel_l2(got[v], exp[v]) <= 1e-11


@pytest.mark.parametrize("component", [0, 4])
@pytest.mark.parametrize("seed", [1, 2])
def test_reach_of_a_nonfinite_cell(cuda_device, component, seed):
    """A NaN cell spoils the faces it belongs to and no other: its limited
    differences do not carry it one face further."""
    q, kxyz, vol = _strong_block((11, 12, 13), seed, 0.5)
    at = (5, 6, 6)
    q[(component,) + at] = np.nan
    bad = ~np.isfinite(_rhs(q, kxyz, vol, "minmod")).all(axis=0)
    exp = np.zeros_like(bad)
    for a in range(3):
        for s in (-1, 0, 1):
            c = list(at)
            c[a] += s
            exp[tuple(c)] = True
    np.testing.assert_array_equal(bad, exp)
