"""The FP64 PCG's two forms, one cooperative launch (the default up to a million
cells) and launch by launch (larger grids, and while kernels are timed), against
the oracle's serial solve after a few iterations: Jacobi and Chebyshev degrees
that end in either buffer, spacings of every row form."""
import numpy as np
import pytest

import les_gb300 as G
import oracle as O

pytestmark = pytest.mark.gpu

SPACINGS = {"pow2": (1 / 16, 1 / 8, 1 / 32), "equal": (0.1, 0.1, 0.1), "different": (0.07, 0.1, 0.03)}


@pytest.mark.parametrize("form", ["cooperative", "launches"])
@pytest.mark.parametrize("h", list(SPACINGS))
@pytest.mark.parametrize("deg", [0, 1, 2, 3, 4, 5], ids=["jacobi"] + ["cheb%d" % d for d in range(1, 6)])
@pytest.mark.parametrize("shape", [(9, 8, 33), (40, 19, 35)], ids=lambda s: "x".join(map(str, s)))
def test_iterate_follows_the_oracle(oracle_lib, shape, deg, h, form):
    rng, om = np.random.default_rng(sum(shape) + deg), O.Mesh(*shape, *SPACINGS[h])
    solid = (rng.random(om.n) < 0.05).astype(np.uint8)
    b, x0 = rng.standard_normal(om.n), rng.standard_normal(om.n)
    A = oracle_lib.build_stencil(om, solid)
    pc, lmin, lmax, cap = (G.PC_CHEBYSHEV if deg else G.PC_JACOBI), 3 * np.pi ** 2, 4 * sum(1 / d ** 2 for d in SPACINGS[h]), 12
    x = x0.copy()
    it, _ = oracle_lib.pcg(om, A, b, x, pc, lmin=lmin, lmax=lmax, degree=max(deg, 1), max_iter=cap, tol=1e-13)
    with G.Context(G.Mesh(*shape, *SPACINGS[h])) as c:
        c.upload_mask(solid)
        c.build_stencil()
        c.upload("b", b)
        c.upload("p", x0)
        if form == "launches":
            c.profile(1)
        st, r = c.pcg(G.pcg_opts(precond=pc, max_iter=cap, tol=1e-13, lambda_min=lmin, lambda_max=lmax, degree=max(deg, 1)))
        got = c.download("p")
        assert ("spmv_f64" in c.profile_all()) == (form == "launches")
    assert st == G.NOT_CONVERGED and r.iters == it == cap
    # the operations are the oracle's; the sums are grouped differently: 24 of them,
    # each within n 2^-53 = 3e-12 relative, and the recurrence's own growth of them
    assert np.max(np.abs(got - x)) < 1e-9 * np.max(np.abs(x))
