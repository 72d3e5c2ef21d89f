"""The FP64 kernels' forms for different spacings -- powers of two, one
spacing that is none, three different ones -- on grids whose edges fall inside
blocks and march chunks: bit-identical to the oracle (up to the sign of zero)."""
import ctypes
import ctypes.util

import numpy as np
import pytest

import les_gb300 as G
import oracle as O

SHAPES = [(5, 4, 4), (9, 8, 33), (12, 17, 31), (40, 9, 65), (70, 33, 32)]
SPACINGS = {"pow2": (1 / 16, 1 / 16, 1 / 16), "pow2_mixed": (1 / 16, 1 / 8, 1 / 32), "equal": (0.1, 0.1, 0.1),
            "yz_equal": (0.07, 0.1, 0.1), "xy_equal": (0.1, 0.1, 0.03), "different": (0.07, 0.1, 0.03)}


def _setup(shape, h, solids, seed=1):
    rng = np.random.default_rng(seed)
    m, om = G.Mesh(*shape, *h), O.Mesh(*shape, *h)
    solid = (rng.random(m.n) < 0.08).astype(np.uint8) if solids else np.zeros(m.n, np.uint8)
    return rng, m, om, solid


@pytest.mark.gpu
@pytest.mark.parametrize("solids", [0, 1])
@pytest.mark.parametrize("h", list(SPACINGS))
@pytest.mark.parametrize("shape", SHAPES)
def test_rows_and_preconditioners(oracle_lib, shape, h, solids):
    rng, m, om, solid = _setup(shape, SPACINGS[h], solids)
    A = oracle_lib.build_stencil(om, solid)
    x = rng.standard_normal(m.n)
    want = np.zeros(m.n)
    oracle_lib.spmv(om, A, x, want)
    with G.Context(m) as c:
        c.upload_mask(solid)
        c.build_stencil()
        c.upload("p", x)
        c.spmv("p", "b")
        assert np.array_equal(c.download("b"), want)
        oracle_lib.jacobi_precond(A, x, want)
        c.precond_apply(G.pcg_opts(precond=G.PC_JACOBI), "p", "b")
        assert np.array_equal(c.download("b"), want)
        lmax = 4 * sum(1 / d ** 2 for d in SPACINGS[h])
        for degree in (1, 2, 4, 5):
            want[:] = 0
            oracle_lib.cheb_apply(om, A, 3 * np.pi ** 2, lmax, degree, x, want)
            c.precond_apply(G.pcg_opts(precond=G.PC_CHEBYSHEV, lambda_min=3 * np.pi ** 2, lambda_max=lmax,
                                       degree=degree), "p", "b")
            assert np.array_equal(c.download("b"), want), degree


def test_division_by_a_constant():
    """q = RN(x y), q + (x - q d) y with y = RN(1/d) is RN(x/d): the device's
    three operations, on the host with the C library's fma."""
    fma = ctypes.CDLL(ctypes.util.find_library("m")).fma
    fma.restype, fma.argtypes = ctypes.c_double, [ctypes.c_double] * 3
    rng = np.random.default_rng(0)
    ds = [6 * 128.0 ** 2, 2 * (1e4 + 1e4 + 1e4), 2 * (1 / 0.07) ** 2, 0.2, 2 / 3, 1e-4, np.nextafter(2.0, 1), np.nextafter(1.0, 2)]
    ds += list(rng.uniform(1, 2, 24))
    for d in ds:
        y = 1.0 / d
        xs = rng.uniform(1, 2, 400) * 2.0 ** rng.integers(-600, 600, 400)
        k = rng.integers(1, 1 << 52, 200) * 2 + 1   # quotients next to a rounding boundary: x = d (k + 1/2) ulp
        xs = np.concatenate([xs, -xs[:100], d * (1 + k * 2.0 ** -53), np.nextafter(d * (1 + k * 2.0 ** -53), 4)])
        for x in xs:
            q = x * y
            assert fma(fma(-q, d, x), y, q) == x / d, (x, d)
