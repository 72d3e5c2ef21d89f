"""The bounded wait of the cooperative FP64 PCG, without a GPU fault."""
import numpy as np
import pytest

import les_gb300 as G

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("deg", [0, 4], ids=["jacobi", "cheb4"])
@pytest.mark.parametrize("shape", [(4, 4, 5), (24, 20, 36)], ids=["one block", "several"])
def test_cooperative_wait_gives_up_and_the_context_recovers(shape, deg):
    """With LES_OPT_TEST_STALL the first block never arrives at the exchange, so
    every block's bounded wait (about 2 s) gives up: LES_TIMEOUT, x as it was, and
    with the option off the same context solves."""
    m = G.Mesh(*shape, 0.1, 0.1, 0.1)
    rng = np.random.default_rng(1)
    b, x0 = rng.standard_normal(m.n), rng.standard_normal(m.n)
    o = G.pcg_opts(precond=G.PC_CHEBYSHEV if deg else G.PC_JACOBI, max_iter=500, tol=1e-8 * np.linalg.norm(b),
                   lambda_min=3 * np.pi ** 2, lambda_max=1200.0, degree=max(deg, 1))
    with G.Context(m) as c:
        c.upload_mask(np.zeros(m.n, np.uint8))
        c.build_stencil()
        c.upload("b", b)
        c.upload("p", x0)
        c.set_option(G.OPT_TEST_STALL, 1)
        with pytest.raises(G.LesError) as e:
            c.pcg(o)
        assert e.value.status == G.TIMEOUT
        assert np.array_equal(c.download("p"), x0)
        c.set_option(G.OPT_TEST_STALL, 0)
        st, r = c.pcg(o)
        assert st == G.OK and r.residual < o.tol
        c.spmv("p", "p_rhs")
        assert np.linalg.norm(b - c.download("p_rhs")) < 2 * o.tol
