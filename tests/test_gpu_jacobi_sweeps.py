"""The stationary Jacobi solver: bit-identical to the oracle, and as many sweeps,
for spacings that take each form of the divisions, with obstacles at the walls
and the outlet, and with tolerances met in different places."""
import numpy as np
import pytest

import les_gb300 as G
import oracle as O

pytestmark = pytest.mark.gpu

SHAPES = [(3, 3, 3), (4, 5, 40), (5, 9, 33), (18, 10, 34), (9, 17, 70)]
SPACINGS = {"equal_pow2": (1 / 16, 1 / 16, 1 / 16), "pow2": (1 / 16, 1 / 8, 1 / 32), "general": (0.05, 0.07, 0.06),
            "equal": (0.01, 0.01, 0.01)}


@pytest.mark.parametrize("h", list(SPACINGS))
@pytest.mark.parametrize("solids", [0, 1])
@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s)))
def test_jacobi_sweeps_match_the_oracle(oracle_lib, shape, solids, h):
    rng = np.random.default_rng(sum(shape))
    m, om = G.Mesh(*shape, *SPACINGS[h]), O.Mesh(*shape, *SPACINGS[h])
    solid = (rng.random(m.n) < 0.15 * solids).astype(np.uint8)
    f = {k: rng.uniform(-1, 1, m.n) for k in ("u", "v", "w", "p")}
    with G.Context(m) as c:
        c.upload_mask(solid)
        for k in "uvw":
            c.upload(k, f[k])
        for sweeps, tol in ((0, 1e-6), (1, 1e-6), (2, 0.0), (33, 0.0), (400, 1e-1), (400, 1e-3)):
            c.upload("p", f["p"])
            got = c.solve_jacobi(1e-2, 1.2, sweeps, tol)
            p = f["p"].copy()
            want = oracle_lib.solve_jacobi(om, 1e-2, 1.2, f["u"], f["v"], f["w"], p, solid, sweeps, tol)
            assert got == want, (sweeps, tol, got, want)
            assert np.array_equal(c.download("p"), p), (sweeps, tol)
