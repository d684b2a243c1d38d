"""Projection and diagnostics on the device against the oracle: the separable
mapping and the fixed-point sine-product + Gaussian solution."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CASES = {
    "curved": dict(n_cells=(3, 4, 2), mesh_type=1, deformation=0.08, ic_params=(0.9, 0.1, 0.45)),
    "curved-box": dict(n_cells=(2, 2, 3), mesh_type=1, deformation=0.06, domain_lo=(-1.0, 0.2, 0.5),
                       domain_hi=(1.0, 0.7, 2.0), velocity=(0.3, -0.7, 0.2), ic_params=(0.0, 0.5, 0.25)),
    "affine": dict(n_cells=(4, 3, 2), ic_params=(0.2, 0.7, 0.0)),
    "wave": dict(n_cells=(3, 2, 2), mesh_type=1, deformation=0.05, initial_condition=2),
    "blob": dict(n_cells=(3, 2, 2), initial_condition=1, ic_params=(0.4, 0.5, 0.6, 0.15)),
}


@pytest.mark.parametrize("degree", [1, 2, 3, 4, 5, 6])
@pytest.mark.parametrize("case", sorted(CASES))
def test_projection_and_diagnostics_match_oracle(cuda, oracle_mod, adv_lib, case, degree):
    cfg = dict(CASES[case], degree=degree)
    o, op = oracle_mod.Oracle(**cfg), adv_lib.AdvectionOperation(**cfg)
    d = op.initialize_dof_vector()
    for t in (0.0, 0.37, 2.5, -1.25):
        op.project_initial(d, t)
        ref = o.project(t)
        # binary64 phases of size |v t| / L and S^-1 (norm at most 4^3 at degree 6)
        assert np.abs(d.cpu().numpy() - ref).max() <= 1e-13 * np.abs(ref).max()
    u = np.random.default_rng(degree).standard_normal(o.n_dofs)
    ud = cuda.from_numpy(u).cuda()
    got, ref = op.l2_error(ud, 0.3), o.l2_error(u, 0.3)
    np.testing.assert_allclose(got, ref, rtol=1e-12)
    np.testing.assert_allclose(op.compute_mass_and_energy(ud), o.mass_energy(u), rtol=1e-12, atol=1e-13)


def test_projection_far_from_the_initial_time(cuda, oracle_mod, adv_lib):
    """Phases beyond the fixed-point range (2^20 turns) in binary64."""
    cfg = dict(CASES["curved"], degree=3)
    o, op = oracle_mod.Oracle(**cfg), adv_lib.AdvectionOperation(**cfg)
    d = op.initialize_dof_vector()
    for t in (1e5, 3e7):
        op.project_initial(d, t)
        ref = o.project(t)
        # the phase v t itself is rounded to 2^-53 of its size, times |d u / d phase| < 10 and S^-1
        assert np.abs(d.cpu().numpy() - ref).max() <= 200 * 2.0 ** -53 * t
