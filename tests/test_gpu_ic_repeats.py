"""The IC(0) apply many times over on a grid of many tiles, where every tile
takes its neighbours' values from other blocks: each apply bit-identical to the
oracle's serial sweeps."""
import numpy as np
import pytest

import les_gb300 as G
import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(12, 35, 97), (24, 66, 40)], ids=lambda s: "x".join(map(str, s)))
def test_repeated_applies(oracle_lib, shape):
    h = (0.05, 0.07, 0.06)
    om = O.Mesh(*shape, *h)
    rng = np.random.default_rng(1)
    solid = np.zeros(om.n, np.uint8)
    A = oracle_lib.build_stencil(om, solid)
    L = oracle_lib.ic_build(om, A)
    with G.Context(G.Mesh(*shape, *h)) as c:
        c.upload_mask(solid)
        c.build_stencil()
        c.build_ic()
        for _ in range(4):
            r, z = rng.standard_normal(om.n), np.zeros(om.n)
            oracle_lib.ic_apply(om, L, r, z)
            c.upload("p", r)
            for n in range(25):
                c.precond_apply(G.pcg_opts(precond=G.PC_IC), "p", "b")
                assert np.array_equal(c.download("b"), z), n
