"""L2 error against the exact solution many periods from the initial time: the
fixed-point solution takes phases below 2^20 turns, binary64 the others."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# turns of the first velocity component (1 over a box of edge 1)
@pytest.mark.parametrize("turns", [1023.75, 2.0 ** 20 - 1.25, 2.0 ** 20 - 0.5, 2.0 ** 20, 2.0 ** 20 + 0.375, 3e7, -1e5,
                                   -(2.0 ** 20) - 0.25])
@pytest.mark.parametrize("curved", [0, 1])
def test_l2_error_far_from_the_initial_time(cuda, oracle_mod, adv_lib, curved, turns):
    cfg = dict(degree=3, n_cells=(3, 4, 2), mesh_type=curved, deformation=0.08 * curved, velocity=(1.0, -0.7, 0.2),
               ic_params=(0.9, 0.1, 0.45))
    o, op = oracle_mod.Oracle(**cfg), adv_lib.AdvectionOperation(**cfg)
    # the solution's own interpolant (the error is that of the mesh) and data of size 1
    for u in (o.project(turns), np.random.default_rng(1).standard_normal(o.n_dofs)):
        got, ref = op.l2_error(cuda.from_numpy(u).cuda(), turns), o.l2_error(u, turns)
        # phases are rounded to 2^-53 of |v t|; |d u / d phase| < 10, in numerator and norm of both sides
        np.testing.assert_allclose(got, ref, rtol=0, atol=400 * 2.0 ** -53 * max(abs(turns), 1.0))
