"""GS-SOR and the IC(0) apply on a grid of more planes than a dimension of a
launch grid holds (65535 blocks): bit-identical to the oracle."""
import numpy as np
import pytest

import les_gb300 as G
import oracle as O

pytestmark = pytest.mark.gpu

SHAPE = (66000, 4, 5)


def test_gs_sweeps(oracle_lib):
    h, rng = (0.05, 0.07, 0.06), np.random.default_rng(2)
    om = O.Mesh(*SHAPE, *h)
    solid = (rng.random(om.n) < 0.02).astype(np.uint8)
    f = {k: rng.uniform(-1, 1, om.n) for k in ("u", "v", "w", "p")}
    with G.Context(G.Mesh(*SHAPE, *h)) as c:
        c.upload_mask(solid)
        for k, a in f.items():
            c.upload(k, a)
        got = c.solve_gs(1e-2, 1.2, 3, 1.5, 0.0)
        p = c.download("p")
    ref = f["p"].copy()
    assert got == oracle_lib.solve_gs(om, 1e-2, 1.2, f["u"], f["v"], f["w"], ref, solid, 3, 1.5, 0.0)
    assert np.array_equal(p, ref)


def test_ic_apply(oracle_lib):
    h, rng = (0.05, 0.07, 0.06), np.random.default_rng(3)
    om = O.Mesh(*SHAPE, *h)
    A = oracle_lib.build_stencil(om, np.zeros(om.n, np.uint8))
    L = oracle_lib.ic_build(om, A)
    r, z = rng.standard_normal(om.n), np.zeros(om.n)
    oracle_lib.ic_apply(om, L, r, z)
    with G.Context(G.Mesh(*SHAPE, *h)) as c:
        c.set_ic_factor(L)
        c.upload("p", r)
        c.precond_apply(G.pcg_opts(precond=G.PC_IC), "p", "b")
        assert np.array_equal(c.download("b"), z)
