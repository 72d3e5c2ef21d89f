"""Adjoints whose pressure solves break down (solid cells in the matrix, a bounded
inner solve): the captured solve ends where the one driven from the host does,
with the same status or the same gradient."""
import numpy as np
import pytest

import les_gb300 as G

pytestmark = pytest.mark.gpu


def _adjoint(dims, h, seed, graph):
    rng, m = np.random.default_rng(seed), G.Mesh(*dims, *h)
    solid = (rng.random(m.n) < 0.1).astype(np.uint8)
    with G.Context(m) as c:
        c.set_option(G.OPT_GRAPH, graph)
        c.upload_mask(solid)
        c.build_stencil()
        for k in ("u", "v", "w", "p"):
            c.upload(k, rng.standard_normal(m.n) * (1 if k == "u" else 0.1))
        prm = G.step_params(nu=1e-5, rho=1.2, cs=0.17, cfl_conv=0.3, cfl_visc=0.2, dt_max=1e-4, dt_fixed=1e-4, rel_tol=1e-6,
                            pcg=G.pcg_opts(precond=G.PC_CHEBYSHEV, max_iter=2000, tol=1e-8, lambda_min=3 * np.pi ** 2,
                                           lambda_max=4 * sum(1 / d ** 2 for d in h), degree=4, precision=G.MIXED,
                                           inner_rtol=1e-4, inner_max_iter=50))
        c.set_inlet(np.ones(dims[1] * dims[2]))
        try:
            j = c.adjoint_forward(prm, 3, 2, (0, dims[0], 0, dims[1], 0, dims[2]), 1e-10)
            grad, gcs = c.adjoint_backward()
            return G.OK, j, np.array(grad), gcs
        except G.LesError as e:
            return e.status, None, None, None


@pytest.mark.parametrize("dims,h", [((20, 12, 9), (0.1, 0.1, 0.1)), ((30, 16, 16), (0.03, 0.025, 0.04))],
                         ids=lambda v: "x".join(map(str, v)))
@pytest.mark.parametrize("seed", [3, 36, 37, 38, 43, 45])
def test_captured_and_host_driven_solves_end_alike(seed, dims, h):
    a, b = _adjoint(dims, h, seed, 1), _adjoint(dims, h, seed, 0)
    assert a[0] == b[0]
    if a[0] == G.OK:
        assert a[1] == b[1] and a[3] == b[3] and np.array_equal(a[2], b[2])
