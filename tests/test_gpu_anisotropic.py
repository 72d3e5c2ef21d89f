"""Mixed Chebyshev solves on cells much longer along i than along j and k: the
iterate after a few inner iterations against the one-kernel-per-operation form,
for ratios on both sides of the line beyond which the scaled levels of the plane
marches and the cluster would leave FP32's range, and right-hand sides whose
squares are near its end."""
import numpy as np
import pytest

import les_gb300 as G

pytestmark = pytest.mark.gpu


def _iterate(shape, h, b, deg, fused):
    m = G.Mesh(*shape, *h)
    with G.Context(m) as c:
        c.set_option(G.OPT_FUSED, fused)
        c.upload_mask(np.zeros(m.n, np.uint8))
        c.build_stencil()
        c.upload("b", b)
        c.upload("p", np.zeros(m.n))
        lmax = 4 * sum(1 / d ** 2 for d in h)
        st, r = c.pcg(G.pcg_opts(precond=G.PC_CHEBYSHEV, max_iter=8, tol=1e-12 * np.linalg.norm(b), lambda_min=lmax / 400,
                                 lambda_max=lmax, degree=deg, precision=G.MIXED, inner_rtol=1e-4))
        return st, r.iters, c.download("p")


@pytest.mark.parametrize("scale", [1.0, 2.0 ** 50])
@pytest.mark.parametrize("deg,ratio", [(7, 8), (7, 12), (7, 1000), (4, 250), (4, 350), (4, 3000), (2, 3000)])
@pytest.mark.parametrize("shape", [(32, 32, 32), (40, 64, 66)], ids=["small", "medium"])
def test_long_cells_follow_unfused(shape, deg, ratio, scale):
    h = (ratio / 32, 1 / 32, 1 / 32)
    b = np.random.default_rng(3).standard_normal(shape)
    b[-1] = 0.0
    b = b.reshape(-1) * scale
    f, u = _iterate(shape, h, b, deg, 1), _iterate(shape, h, b, deg, 0)
    assert f[:2] == u[:2] == (G.NOT_CONVERGED, 8)
    # eight FP32 iterations, each within some FP32 roundings of the other form
    assert np.max(np.abs(f[2] - u[2])) < 1e-4 * np.max(np.abs(u[2]))
