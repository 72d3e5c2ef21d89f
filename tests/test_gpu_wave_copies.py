"""GS-SOR and the IC(0) applies on the fields' own arrays, without copies of the
operands (LES_OPT_WAVE_COPIES 0): bit-identical to the oracle and to the form
with copies; and what the copies leave allocated."""
import numpy as np
import pytest
import torch

import les_gb300 as G
import oracle as O

pytestmark = pytest.mark.gpu

SHAPES = [(3, 3, 3), (4, 6, 40), (9, 7, 35), (40, 5, 34), (34, 19, 66), (130, 12, 36)]
SPACINGS = {"pow2": (1 / 16, 1 / 8, 1 / 32), "general": (0.05, 0.07, 0.06)}


def _context(shape, h, copies):
    c = G.Context(G.Mesh(*shape, *h))
    c.set_option(G.OPT_WAVE_COPIES, copies)
    return c


@pytest.mark.parametrize("h", list(SPACINGS))
@pytest.mark.parametrize("solids", [0.0, 0.15])
@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s)))
def test_gs_without_copies(oracle_lib, shape, solids, h):
    rng, om = np.random.default_rng(sum(shape)), O.Mesh(*shape, *SPACINGS[h])
    solid = (rng.random(om.n) < solids).astype(np.uint8)
    f = {k: rng.uniform(-1, 1, om.n) for k in ("u", "v", "w", "p")}
    with _context(shape, SPACINGS[h], 0) as c:
        c.upload_mask(solid)
        for k in "uvw":
            c.upload(k, f[k])
        for sweeps, tol in ((1, 0.0), (2, 0.0), (17, 0.0), (200, 1e-1)):
            c.upload("p", f["p"])
            ref = f["p"].copy()
            got = c.solve_gs(1e-2, 1.2, sweeps, 1.4, tol)
            assert got == oracle_lib.solve_gs(om, 1e-2, 1.2, f["u"], f["v"], f["w"], ref, solid, sweeps, 1.4, tol)
            assert np.array_equal(c.download("p"), ref), (sweeps, tol)


@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s)))
def test_ic_without_copies(oracle_lib, shape):
    h = SPACINGS["general"]
    rng, om = np.random.default_rng(sum(shape)), O.Mesh(*shape, *h)
    solid = (rng.random(om.n) < 0.1).astype(np.uint8)
    A = oracle_lib.build_stencil(om, solid)
    L = oracle_lib.ic_build(om, A)
    r, z = rng.standard_normal(om.n), np.zeros(om.n)
    p = {}
    for copies in (0, 1):
        with _context(shape, h, copies) as c:
            c.upload_mask(solid)
            c.build_stencil()
            c.build_ic()
            c.upload("p", r)
            for pc, M in ((G.PC_IC, L), (G.PC_IC_A, A)):
                c.precond_apply(G.pcg_opts(precond=pc), "p", "b")
                oracle_lib.ic_apply(om, M, r, z)
                assert np.array_equal(c.download("b"), z, equal_nan=True), pc
            for precision in (G.FP64, G.MIXED):
                c.upload("b", r)
                c.upload("p", np.zeros(om.n))
                st, res = c.pcg(G.pcg_opts(precond=G.PC_IC, max_iter=6, tol=1e-30, precision=precision, inner_rtol=1e-4))
                p[copies, precision] = (st, res.iters, c.download("p"))
    for precision in (G.FP64, G.MIXED):   # the same applies in the same order
        a, b = p[0, precision], p[1, precision]
        assert a[:2] == b[:2] and np.array_equal(a[2], b[2], equal_nan=True)


def test_what_the_copies_leave_allocated():
    """Small copies stay, large ones (1.2 GB here) are given back at the end of the
    apply, and without copies nothing is allocated."""
    def left(shape, copies):
        with _context(shape, (0.05,) * 3, copies) as c:
            c.upload_mask(np.zeros(c.n, np.uint8))
            c.build_stencil()
            c.build_ic()
            c.set_option(G.OPT_WAVE_COPIES, 0)
            c.precond_apply(G.pcg_opts(precond=G.PC_IC), "p", "b")   # everything else is allocated
            c.set_option(G.OPT_WAVE_COPIES, copies)
            before = torch.cuda.mem_get_info()[0]
            c.precond_apply(G.pcg_opts(precond=G.PC_IC), "p", "b")
            return before - torch.cuda.mem_get_info()[0]

    left((9, 7, 35), 1)   # loads the kernels of both forms
    assert left((64, 400, 400), 1) == 0
    assert left((96, 64, 64), 0) == 0
    assert 0 < left((96, 64, 64), 1) < (48 << 20)   # 9 arrays of 16 x 2 tiles, 130 steps, 128 cells: 38 MB
