"""The FP32 face flux's clamped minmod and its reciprocals and roots of normal
arguments, at the states where they could go wrong: strong jumps and sign changes
in every direction, equal and vanishing differences, tiny normals.

Tolerance: relative L2 <= 1e-5 of the inviscid right-hand side against the FP64
oracle.  With jumps of the size of the state the face differences are as large
as the fluxes, so the error is the fluxes' own: about 50 FP32 roundings of 6e-8.
"""
import numpy as np
import pytest

from famrdp_jax_b200.core.types import Metrics
from famrdp_jax_b200.rhs.invscd import compute_invscd_rhs
from oracle.ref import NP
from parity_util import dev, host, random_block, rel_l2

pytestmark = pytest.mark.gpu


def _both(q, kxyz, vol, limiter):
    m = Metrics(jac=dev(vol), kxyz=dev(kxyz), vol=dev(vol))
    got = host(compute_invscd_rhs(dev(q), m, ghost=2, gamma=1.4, reconstruct="muscl2", flux="roe", limiter=limiter,
                                  precision="f32"))
    return got, NP.compute_invscd_rhs(q, kxyz, vol, ghost=2, gamma=1.4, limiter=limiter)


def _state(shape, seed, mach, levels):
    """Jumps of up to a factor of 20; with ``levels`` the values are few, so that
    neighbouring differences are often equal, opposite or zero."""
    rng = np.random.default_rng(seed)
    pick = (lambda: rng.integers(0, levels, shape) / levels) if levels else (lambda: rng.random(shape))
    rho, p = np.exp(3.0 * pick() - 1.5), np.exp(3.0 * pick() - 1.5)
    u, v, w = (mach * (2.0 * pick() - 1.0) for _ in range(3))
    return np.stack([rho, rho * u, rho * v, rho * w, p / 0.4 + 0.5 * rho * (u * u + v * v + w * w)])


@pytest.mark.parametrize("limiter", ["minmod", "vanleer"])
@pytest.mark.parametrize("shape,mach,levels", [((5, 5, 5), 1.0, 0), ((9, 12, 35), 0.05, 2), ((6, 31, 64), 3.0, 4)])
def test_strong_jumps(cuda_device, shape, mach, levels, limiter):
    _, kxyz, vol = random_block(shape, 7)
    got, exp = _both(_state(shape, 11, mach, levels), kxyz, vol, limiter)
    for v in range(5):
        assert rel_l2(got[v], exp[v]) <= 1e-5


@pytest.mark.parametrize("scale", [1e-12, 1e8])
def test_scaled_normals(cuda_device, scale):
    _, kxyz, vol = random_block((7, 9, 33), 8)
    got, exp = _both(_state((7, 9, 33), 12, 0.5, 0), kxyz * scale, vol, "minmod")
    for v in range(5):
        assert rel_l2(got[v], exp[v]) <= 1e-5
