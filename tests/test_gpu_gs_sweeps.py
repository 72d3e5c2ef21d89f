"""GS-SOR with sweeps in flight: bit-identical to the oracle's serial sweeps, and
the same number of them, on grids of one and several tiles with ragged edges,
with solid cells at the walls, the inlet and the outlet, and with tolerances
that are met in the middle of a batch of sweeps."""
import numpy as np
import pytest

import les_gb300 as G
import oracle as O

pytestmark = pytest.mark.gpu

SHAPES = [(3, 3, 3), (4, 5, 40), (9, 7, 35), (33, 6, 34), (34, 19, 66), (70, 11, 9), (40, 37, 70), (130, 12, 36)]
SPACINGS = {"equal_pow2": (1 / 16, 1 / 16, 1 / 16), "pow2": (1 / 16, 1 / 8, 1 / 32), "general": (0.05, 0.07, 0.06)}


def _case(shape, h, solids, seed):
    rng = np.random.default_rng(seed)
    n = int(np.prod(shape))
    solid = np.zeros(shape, np.uint8)
    if solids == "random":
        solid[rng.random(shape) < 0.15] = 1
    elif solids == "box":
        a = [max(1, s // 3) for s in shape]
        solid[a[0]:, a[1]:2 * a[1] + 1, :a[2] + 1] = 1   # reaches the outlet and a wall
    f = {k: rng.uniform(-1, 1, n) for k in ("u", "v", "w", "p")}
    return O.Mesh(*shape, *h), solid.reshape(-1), f


def _both(oracle_lib, om, solid, f, sweeps, tol, omega=1.7):
    with G.Context(G.Mesh(om.nx, om.ny, om.nz, om.dx, om.dy, om.dz)) as c:
        c.upload_mask(solid)
        for k, a in f.items():
            c.upload(k, a)
        got = c.solve_gs(1e-2, 1.2, sweeps, omega, tol)
        p = c.download("p")
    ref = f["p"].copy()
    want = oracle_lib.solve_gs(om, 1e-2, 1.2, f["u"], f["v"], f["w"], ref, solid, sweeps, omega, tol)
    return got, want, p, ref


@pytest.mark.parametrize("h", list(SPACINGS))
@pytest.mark.parametrize("solids", ["none", "random", "box"])
@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s)))
def test_sweeps_in_flight_match_serial_sweeps(oracle_lib, shape, solids, h):
    om, solid, f = _case(shape, SPACINGS[h], solids, sum(shape))
    for sweeps in (1, 2, 3, 40):
        got, want, p, ref = _both(oracle_lib, om, solid, f, sweeps, 0.0)
        assert got == want
        assert np.array_equal(p, ref), (sweeps, np.flatnonzero(p != ref)[:5])


@pytest.mark.parametrize("solids", ["none", "box"])
def test_tolerance_met_inside_a_batch(oracle_lib, solids):
    om, solid, f = _case((20, 9, 38), SPACINGS["general"], solids, 5)
    seen = set()
    for tol in (1e2, 1.0, 1e-1, 1e-2, 1e-4, 1e-6, 1e-9):
        got, want, p, ref = _both(oracle_lib, om, solid, f, 300, tol, 1.2)
        assert got == want, (tol, got, want)
        assert np.array_equal(p, ref), tol
        seen.add(got)
    if solids == "none":   # (the box case does not converge)
        assert len(seen) >= 4   # different places in different batches
