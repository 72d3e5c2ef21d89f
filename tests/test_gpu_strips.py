"""The register-column strips of a solve with a forced strip shape (batched
ensembles run them too) on rows that end around a tile's edge: the iterate after
a few inner iterations against the one-kernel-per-operation form, and the
kernels compiled for a row stride against those that read it at run time."""
import numpy as np
import pytest

import les_gb300 as G

pytestmark = pytest.mark.gpu

H = (0.03, 0.025, 0.04)
PCS = [(G.PC_JACOBI, 0)] + [(G.PC_CHEBYSHEV, d) for d in (2, 3, 4, 5, 6, 7)]
IDS = ["jacobi", "cheb2", "cheb3", "cheb4", "cheb5", "cheb6", "cheb7"]


def _iterate(shape, pc, deg, options, cap=8):
    m = G.Mesh(*shape, *H)
    b = np.random.default_rng(sum(shape)).standard_normal(shape)
    b[-1] = 0.0
    b = b.reshape(-1)
    with G.Context(m) as c:
        for opt, v in options:
            c.set_option(opt, v)
        c.upload_mask(np.zeros(m.n, np.uint8))
        c.build_stencil()
        c.upload("b", b)
        c.upload("p", np.zeros(m.n))
        st, r = c.pcg(G.pcg_opts(precond=pc, max_iter=cap, tol=1e-12 * np.linalg.norm(b), lambda_min=3 * np.pi ** 2,
                                 lambda_max=4 * sum(1 / d ** 2 for d in H), degree=max(deg, 1), precision=G.MIXED,
                                 inner_rtol=1e-4))
        return st, r.iters, c.download("p")


def _strips(pc, deg):
    return [(G.OPT_ROWS_A, 8), (G.OPT_ROWS_B, 16 if pc == G.PC_JACOBI else (8 if deg <= 4 else 4))]


# a tile owns 32 - S cells at a wall and 32 - 2 S between (S levels): one tile, two,
# and one more, each by its last cell
def _lengths(deg):
    S = max(deg - 1, 1)
    two, three = 2 * (32 - S), 2 * (32 - S) + 32 - 2 * S
    return sorted({14, 31, 32, 33, two - 1, two, two + 1, three, three + 1, 130, 257})


@pytest.mark.parametrize("pc,deg,nz", [(pc, deg, nz) for pc, deg in PCS for nz in _lengths(deg)],
                         ids=lambda v: str(v))
def test_strips_follow_unfused(pc, deg, nz):
    shape = (17, 14 + 5 * (nz % 3), nz)   # row strips end evenly and not
    f, u = _iterate(shape, pc, deg, _strips(pc, deg)), _iterate(shape, pc, deg, [(G.OPT_FUSED, 0)])
    assert f[:2] == u[:2] == (G.NOT_CONVERGED, 8)
    # eight FP32 iterations, each within some FP32 roundings of the other form
    assert np.max(np.abs(f[2] - u[2])) < 1e-4 * np.max(np.abs(u[2]))


@pytest.mark.parametrize("pc,deg", PCS, ids=IDS)
@pytest.mark.parametrize("nz", [32, 64, 128, 256])
def test_strips_of_a_compiled_stride(nz, pc, deg):
    """The same arithmetic in the same order: the same bits."""
    strips = _strips(pc, deg)
    a = _iterate((20, 21, nz), pc, deg, strips + [(G.OPT_COL_STRIDE, 1)], 20)
    b = _iterate((20, 21, nz), pc, deg, strips + [(G.OPT_COL_STRIDE, 0)], 20)
    assert a[:2] == b[:2] and np.array_equal(a[2], b[2])


@pytest.mark.parametrize("cap", [1, 2, 7])
@pytest.mark.parametrize("pc,deg", [(G.PC_JACOBI, 0), (G.PC_CHEBYSHEV, 4)], ids=["jacobi", "cheb4"])
def test_strips_stop_at_the_iteration_cap(pc, deg, cap):
    f = _iterate((24, 20, 34), pc, deg, _strips(pc, deg), cap)
    assert f[:2] == (G.NOT_CONVERGED, cap) and np.all(np.isfinite(f[2]))
