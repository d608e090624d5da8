"""The FP64 reciprocals and roots of fj_physics.cuh against extended precision
(NumPy's 80-bit long double), at every exponent from -1020 to 1000 with random
mantissas, at powers of two and their neighbours, and at the clamps' values.

2^-53 is half a unit in the last place at worst:
rcp_normal and rcp_any round the result of an exact-residual step once (<= 1.02 of
2^-53, the second-order remainder 1e-18 included), sqrt_normal likewise (<= 1.02),
rsqrt_normal's residual has one rounded product more, halved (<= 1.6 + the final
rounding's share: <= 2.05).
"""
import ctypes
import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest
import torch

from parity_util import dev, host

LD = np.longdouble
pytestmark = [pytest.mark.gpu,
              pytest.mark.skipif(np.finfo(LD).nmant < 63, reason="long double is no wider than double")]

ROOT = Path(__file__).resolve().parent


@pytest.fixture(scope="module")
def roots(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    so = tmp_path_factory.mktemp("roots") / "libroots.so"
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-shared", "-Xcompiler",
                    "-fPIC", "--expt-relaxed-constexpr", "-cudart", "static", "-I",
                    str(ROOT.parent / "famrdp_jax_b200" / "csrc"), str(ROOT / "cuda_f64_roots.cu"), "-o", str(so)],
                   check=True)
    fn = ctypes.CDLL(str(so)).f64_roots
    fn.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_int, ctypes.c_void_p]

    def call(x):
        xd = dev(x)
        out = torch.empty((4, x.size), dtype=torch.float64, device="cuda")
        assert fn(xd.data_ptr(), out.data_ptr(), x.size, torch.cuda.current_stream().cuda_stream) == 0
        return host(out)
    return call


def test_reciprocals_and_roots(cuda_device, roots):
    rng = np.random.default_rng(1)
    ex = np.repeat(np.arange(-1020, 1000), 2000)
    x = np.ldexp(1.0 + rng.random(ex.size), ex)
    x = np.concatenate([x, np.ldexp(1.0, np.arange(-1020, 1001)), np.nextafter(np.ldexp(1.0, np.arange(-1019, 1001)), 0),
                        [1e-300, 1e-30, 1e-150, 1.0 + 1e-300]])
    got, xl = roots(x), x.astype(LD)
    exact = {"rcp": 1 / xl, "rsqrt": 1 / np.sqrt(xl), "sqrt": np.sqrt(xl), "any": 1 / xl}
    for g, (name, bound) in zip(got, (("rcp", 1.02), ("rsqrt", 2.05), ("sqrt", 1.02), ("any", 1.02))):
        err = float(np.abs((g.astype(LD) - exact[name]) / exact[name]).max()) * 2.0 ** 53
        print(f"{name}: {err:.4f} x 2^-53")
        assert err <= bound, name


def test_reciprocal_of_anything(cuda_device, roots):
    x = np.array([0.0, -0.0, np.inf, -np.inf, np.nan, -3.0, 1.5e308])
    got = roots(x)[3]
    with np.errstate(divide="ignore"):
        exp = 1.0 / x
    exp[6] = 0.0  # below the normal range
    np.testing.assert_array_equal(got[:5], exp[:5])
    np.testing.assert_allclose(got[5:], exp[5:], rtol=1.2e-16)
