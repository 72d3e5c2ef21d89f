"""The IC(0) apply on grids of one and several tiles with ragged edges, with the
factor and with the matrix in its place: bit-identical to the oracle's serial
sweeps, and one factor after the other on the same context."""
import numpy as np
import pytest

import les_gb300 as G
import oracle as O

pytestmark = pytest.mark.gpu

SHAPES = [(3, 3, 3), (4, 6, 40), (9, 7, 35), (40, 5, 34), (34, 19, 66), (70, 18, 33), (12, 35, 97)]


@pytest.mark.parametrize("h", [(1 / 16, 1 / 16, 1 / 16), (0.05, 0.07, 0.06)], ids=["pow2", "general"])
@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s)))
def test_ic_apply_on_ragged_tiles(oracle_lib, shape, h):
    rng = np.random.default_rng(sum(shape))
    om = O.Mesh(*shape, *h)
    solid = (rng.random(om.n) < 0.1).astype(np.uint8)
    r, z = rng.standard_normal(om.n), np.zeros(om.n)
    A = oracle_lib.build_stencil(om, solid)
    L = oracle_lib.ic_build(om, A)
    with G.Context(G.Mesh(*shape, *h)) as c:
        c.upload_mask(solid)
        c.build_stencil()
        c.build_ic()
        c.upload("p", r)
        for pc, M in ((G.PC_IC, L), (G.PC_IC_A, A), (G.PC_IC, L)):
            c.precond_apply(G.pcg_opts(precond=pc), "p", "b")
            oracle_lib.ic_apply(om, M, r, z)
            assert np.array_equal(c.download("b"), z, equal_nan=True), pc
