"""Infinities and NaN in the vector of an FP64 matrix product and preconditioner
apply: where the oracle's rows are not finite, ours are not, in every row form --
identity rows (solid cells, the outlet) too, whose zero coefficients meet them."""
import numpy as np
import pytest

import les_gb300 as G
import oracle as O

pytestmark = pytest.mark.gpu

SPACINGS = {"pow2": (1 / 16, 1 / 8, 1 / 32), "equal": (0.1, 0.1, 0.1), "different": (0.07, 0.1, 0.03)}


@pytest.mark.parametrize("bad", [np.inf, -np.inf, np.nan])
@pytest.mark.parametrize("solids", [0.0, 0.1])
@pytest.mark.parametrize("h", list(SPACINGS))
def test_rows(oracle_lib, h, solids, bad):
    shape = (18, 10, 35)
    rng, om = np.random.default_rng(11), O.Mesh(*shape, *SPACINGS[h])
    solid = (rng.random(om.n) < solids).astype(np.uint8)
    A = oracle_lib.build_stencil(om, solid)
    x = rng.standard_normal(om.n)
    x[rng.integers(0, om.n, 12)] = bad
    x.reshape(shape)[-2, 4, 7] = x.reshape(shape)[-1, 3, 20] = bad   # next to the outlet, and in it
    want = np.zeros(om.n)
    with G.Context(G.Mesh(*shape, *SPACINGS[h])) as c:
        c.upload_mask(solid)
        c.build_stencil()
        c.upload("p", x)
        c.spmv("p", "b")
        oracle_lib.spmv(om, A, x, want)
        assert np.array_equal(c.download("b"), want, equal_nan=True)
        oracle_lib.jacobi_precond(A, x, want)
        c.precond_apply(G.pcg_opts(precond=G.PC_JACOBI), "p", "b")
        assert np.array_equal(c.download("b"), want, equal_nan=True)
        for degree in (2, 4):
            want[:] = 0
            lmax = 4 * sum(1 / d ** 2 for d in SPACINGS[h])
            oracle_lib.cheb_apply(om, A, 3 * np.pi ** 2, lmax, degree, x, want)
            c.precond_apply(G.pcg_opts(precond=G.PC_CHEBYSHEV, lambda_min=3 * np.pi ** 2, lambda_max=lmax,
                                       degree=degree), "p", "b")
            assert np.array_equal(c.download("b"), want, equal_nan=True), degree


def test_quotients_of_zeros_keep_their_sign(oracle_lib):
    """The Jacobi preconditioner's division by a constant: +-0 / A_c is +-0, and
    subnormals and the largest numbers take the division."""
    shape, h = (6, 7, 33), (0.07, 0.1, 0.03)
    om = O.Mesh(*shape, *h)
    A = oracle_lib.build_stencil(om, np.zeros(om.n, np.uint8))
    x = np.resize([0.0, -0.0, 1.0, -1.5, 5e-324, -1e-310, 1.7e308, -3e-300, 1e250, np.inf, -np.inf, np.nan], om.n)
    want = np.zeros(om.n)
    oracle_lib.jacobi_precond(A, x, want)
    with G.Context(G.Mesh(*shape, *h)) as c:
        c.upload_mask(np.zeros(om.n, np.uint8))
        c.build_stencil()
        c.upload("p", x)
        c.precond_apply(G.pcg_opts(precond=G.PC_JACOBI), "p", "b")
        got = c.download("b")
    assert np.array_equal(got, want, equal_nan=True)
    number = ~np.isnan(want)
    assert np.array_equal(np.signbit(got[number]), np.signbit(want[number]))
