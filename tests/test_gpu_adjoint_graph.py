"""The adjoint's mixed solves as graph launches against solves driven from the
host: the same kernels in the same order, so the same gradient to the bit (a
grid of the plane marches; the FP32 iteration is deterministic)."""
import numpy as np
import pytest

import les_cases
import les_gb300 as G

pytestmark = pytest.mark.gpu


def _gradient(pc, deg, graph):
    shape, h = (88, 44, 40), 1.0 / 44
    with G.Context(G.Mesh(*shape, h, h, h)) as c:
        c.set_option(G.OPT_GRAPH, graph)
        c.upload_mask(np.zeros(c.n, np.uint8))
        c.build_stencil()
        lmax = c.lambda_max(20)
        solid = les_cases.box_mask(shape, (20, 30, 16, 26, 14, 24))
        f = les_cases.init_fields(shape, 0.02, 3)
        les_cases.velocity_bcs_np(shape, f, solid)
        c.upload_mask(solid)
        c.upload_fields(f)
        c.set_inlet(np.ones(shape[1:]).reshape(-1))
        prm = G.step_params(nu=1e-5, rho=1.2, cs=0.17, cfl_conv=0.3, dt_fixed=1e-4,
                            pcg=G.pcg_opts(precond=pc, max_iter=20000, lambda_min=3 * np.pi ** 2, lambda_max=lmax,
                                           degree=deg, precision=G.MIXED, inner_rtol=1e-4))
        j = c.adjoint_forward(prm, 3, 2, (60, 70, 10, 30, 10, 30), 1e-10)
        grad, gcs = c.adjoint_backward()
        return j, np.array(grad), gcs


@pytest.mark.parametrize("pc,deg", [(G.PC_JACOBI, 1), (G.PC_CHEBYSHEV, 4)], ids=["jacobi", "cheb4"])
def test_graph_solves_match_host_driven(pc, deg):
    a, b = _gradient(pc, deg, 1), _gradient(pc, deg, 0)
    assert a[0] == b[0] and a[2] == b[2]
    assert np.array_equal(a[1], b[1])
