"""The most sweeps that a GS-SOR solve may be asked for: 2^29 progress values,
nx + 34 of them per sweep.  (The solves end after the first sweep.)"""
import numpy as np
import pytest

import les_gb300 as G
import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("copies", [0, 1])
def test_most_sweeps(oracle_lib, copies):
    shape, h = (5, 6, 7), (0.05, 0.07, 0.06)
    om, rng = O.Mesh(*shape, *h), np.random.default_rng(4)
    f = {k: rng.uniform(-1, 1, om.n) for k in ("u", "v", "w", "p")}
    solid, most = np.zeros(om.n, np.uint8), 2 ** 29 // (5 + 34)
    with G.Context(G.Mesh(*shape, *h)) as c:
        c.set_option(G.OPT_WAVE_COPIES, copies)
        for k, a in f.items():
            c.upload(k, a)
        for _ in range(3):   # (the counters start again when their range ends)
            c.upload("p", f["p"])
            assert c.solve_gs(1e-2, 1.2, most, 1.5, 1e300) == 1
            ref = f["p"].copy()
            assert oracle_lib.solve_gs(om, 1e-2, 1.2, f["u"], f["v"], f["w"], ref, solid, most, 1.5, 1e300) == 1
            assert np.array_equal(c.download("p"), ref)
        with pytest.raises(G.LesError) as e:
            c.solve_gs(1e-2, 1.2, most + 1, 1.5, 1e300)
        assert e.value.status == G.BAD_ARG
