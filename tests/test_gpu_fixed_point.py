"""Block fixed-point stages of the FP64 operator (collocation form) against the oracle.

The scale of a cell's block adapts to its data, so a step commutes with any
power of two, cells of very different magnitude sit side by side, and cells
outside the window of exponents (here 2^-400 .. 2^600, infinities, NaN) take
the binary64 path.  Bars: the repository's FP64 bar, 1e-12 of the largest
entry; the fixed-point error is a few 2^-57 of a cell's largest intermediate
value per contraction, below binary64's own rounding.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = 1e-12

# uniform, curved with upwind traces, curved reading every trace, boundary data
MESHES = {
    "uniform": dict(n_cells=(3, 2, 5)),
    "curved": dict(n_cells=(3, 3, 2), mesh_type=1, deformation=0.07),
    "curved-lax-friedrichs": dict(n_cells=(2, 3, 3), mesh_type=1, deformation=0.06, flux_alpha=0.5),
    "curved-dirichlet": dict(n_cells=(2, 3, 2), mesh_type=1, deformation=0.06, periodic=0, initial_condition=2),
    "rotating": dict(n_cells=(2, 2, 3), periodic=0, velocity_type=1, velocity=(1.0, 1.0, 0.3), velocity_period=0.5,
                     initial_condition=1, ic_params=(0.3, 0.5, 0.5, 0.1), boundary_value=0),
}


def gpu_step(torch, adv, cfg, u0, t, dt, steps=1, scheme=None, **kw):
    op = adv.AdvectionOperation(**cfg, **kw)
    u = torch.from_numpy(np.ascontiguousarray(u0)).cuda()
    r, k = op.initialize_dof_vector(), op.initialize_dof_vector()
    op.lsrk_steps(adv.LSRK_5_4 if scheme is None else scheme, t, dt, steps, u, r, k)
    return u.cpu().numpy()


def oracle_step(oracle_mod, cfg, u0, t, dt):
    o = oracle_mod.Oracle(**cfg)
    u, r, k = u0.copy(), np.zeros_like(u0), np.zeros_like(u0)
    o.lsrk_step(t, dt, u, r, k)
    return u


@pytest.mark.parametrize("degree", [1, 2, 3, 4, 5, 6])
@pytest.mark.parametrize("mesh", sorted(MESHES))
def test_step_matches_oracle(cuda, oracle_mod, adv_lib, mesh, degree):
    cfg = dict(MESHES[mesh], degree=degree)
    u0 = np.random.default_rng(degree).standard_normal(oracle_mod.Oracle(**cfg).n_dofs)
    ref = oracle_step(oracle_mod, cfg, u0, 0.1, 0.004)
    for form in (adv_lib.FORM_AUTO, adv_lib.FORM_COLLOCATION_NO_TRACES):
        got = gpu_step(cuda, adv_lib, cfg, u0, 0.1, 0.004, fused_form=form)
        assert np.abs(got - ref).max() <= TOL * np.abs(ref).max(), (mesh, degree, form)


# inside the window, at its lower and upper side, and outside both ends
@pytest.mark.parametrize("exponent", [-900, -450, -300, 300, 620, 900])
@pytest.mark.parametrize("mesh", ["uniform", "curved"])
def test_step_commutes_with_powers_of_two(cuda, oracle_mod, adv_lib, mesh, exponent):
    cfg = dict(MESHES[mesh], degree=3)
    u0 = np.random.default_rng(3).standard_normal(oracle_mod.Oracle(**cfg).n_dofs)
    ref = oracle_step(oracle_mod, cfg, u0, 0.0, 0.004)
    got = np.ldexp(gpu_step(cuda, adv_lib, cfg, np.ldexp(u0, exponent), 0.0, 0.004), -exponent)
    assert np.abs(got - ref).max() <= TOL * np.abs(ref).max()


@pytest.mark.parametrize("mesh", ["uniform", "curved"])
def test_cells_of_different_magnitude(cuda, oracle_mod, adv_lib, mesh):
    """Cells of 2^-470 and of 0 beside cells of 1: a large neighbour's flux
    sets the scale of a small cell, and a cell alone in a small neighbourhood
    takes the binary64 path."""
    cfg = dict(MESHES[mesh], degree=4, n_cells=(6, 5, 4))
    o = oracle_mod.Oracle(**cfg)
    rng = np.random.default_rng(5)
    u0 = rng.standard_normal(o.n_dofs).reshape(-1, 125)
    u0[::7] = 0.0
    u0[40:100] *= 2.0 ** -470
    u0 = u0.reshape(-1)
    ref = oracle_step(oracle_mod, cfg, u0, 0.0, 0.002)
    got = gpu_step(cuda, adv_lib, cfg, u0, 0.0, 0.002)
    assert np.abs(got - ref).max() <= TOL * np.abs(ref).max()
    assert np.abs(got - gpu_step(cuda, adv_lib, cfg, u0, 0.0, 0.002,
                                 fused_form=adv_lib.FORM_COLLOCATION_NO_TRACES)).max() == 0.0


@pytest.mark.parametrize("value", [np.nan, np.inf])
def test_values_that_are_not_finite_stay_local(cuda, oracle_mod, adv_lib, value):
    cfg = dict(MESHES["curved"], degree=4, n_cells=(9, 4, 4))
    n = oracle_mod.Oracle(**cfg).n_dofs
    u0 = np.random.default_rng(6).standard_normal(n)
    clean = gpu_step(cuda, adv_lib, cfg, u0, 0.0, 0.002, scheme=adv_lib.LSRK_3_3).reshape(4, 4, 9, 125)
    u0[(2 + 9 * (1 + 4 * 1)) * 125 + 62] = value
    got = gpu_step(cuda, adv_lib, cfg, u0, 0.0, 0.002, scheme=adv_lib.LSRK_3_3).reshape(4, 4, 9, 125)
    assert not np.isfinite(got[1, 1, 2]).any()
    # three stages reach at most three cells
    np.testing.assert_array_equal(got[:, :, 6:8], clean[:, :, 6:8])


# ---- nodal kernel (apply, perform_stage, vmult)


@pytest.mark.parametrize("degree", [1, 2, 3, 4, 5, 6])
@pytest.mark.parametrize("mesh", sorted(MESHES))
def test_apply_and_vmult_match_oracle(cuda, oracle_mod, adv_lib, mesh, degree):
    cfg = dict(MESHES[mesh], degree=degree)
    o, op = oracle_mod.Oracle(**cfg), adv_lib.AdvectionOperation(**cfg)
    src = np.random.default_rng(20 + degree).standard_normal(o.n_dofs)
    s, d = cuda.from_numpy(src).cuda(), op.initialize_dof_vector()
    op.apply(s, d, 0.1)
    ref = o.apply(src, 0.1)
    assert np.abs(d.cpu().numpy() - ref).max() <= TOL * np.abs(ref).max()
    # weak form: c M u - L u = M (c u - M^{-1} L u)
    op.vmult(s, d, 3.0, 0.1)
    e = op.initialize_dof_vector()
    op.apply_mass(cuda.from_numpy(3.0 * src - ref).cuda(), e)
    e = e.cpu().numpy()
    assert np.abs(d.cpu().numpy() - e).max() <= TOL * np.abs(e).max()


@pytest.mark.parametrize("exponent", [-900, -450, -300, 300, 620, 900])
@pytest.mark.parametrize("mesh", ["uniform", "curved"])
def test_apply_commutes_with_powers_of_two(cuda, oracle_mod, adv_lib, mesh, exponent):
    cfg = dict(MESHES[mesh], degree=5)
    o, op = oracle_mod.Oracle(**cfg), adv_lib.AdvectionOperation(**cfg)
    src = np.random.default_rng(9).standard_normal(o.n_dofs)
    s, d = cuda.from_numpy(np.ldexp(src, exponent)).cuda(), op.initialize_dof_vector()
    op.apply(s, d, 0.0)
    ref = o.apply(src, 0.0)
    assert np.abs(np.ldexp(d.cpu().numpy(), -exponent) - ref).max() <= TOL * np.abs(ref).max()


@pytest.mark.parametrize("mesh", ["uniform", "curved"])
def test_apply_on_cells_of_different_magnitude(cuda, oracle_mod, adv_lib, mesh):
    cfg = dict(MESHES[mesh], degree=4, n_cells=(6, 5, 4))
    o, op = oracle_mod.Oracle(**cfg), adv_lib.AdvectionOperation(**cfg)
    src = np.random.default_rng(8).standard_normal(o.n_dofs).reshape(-1, 125)
    src[::7] = 0.0
    src[20:90] *= 2.0 ** -470  # some with neighbours of 1, some among their like
    src = src.reshape(-1)
    s, d = cuda.from_numpy(src).cuda(), op.initialize_dof_vector()
    op.apply(s, d, 0.0)
    ref, got = o.apply(src, 0.0), d.cpu().numpy()
    assert np.abs(got - ref).max() <= TOL * np.abs(ref).max()
    small = np.abs(ref).reshape(-1, 125).max(axis=1) < 2.0 ** -400  # cells that see no value of 1
    small = np.repeat(small, 125)
    assert small.any()
    assert np.abs(got - ref)[small].max() <= TOL * np.abs(ref[small]).max()
    # one value that is not finite reaches its own cell and the face neighbours
    src[62 + 125 * 40] = np.nan
    op.apply(cuda.from_numpy(src).cuda(), d, 0.0)
    bad = ~np.isfinite(d.cpu().numpy()).reshape(-1, 125).all(axis=1)
    assert bad[40] and bad.sum() <= 7
    keep = np.repeat(~bad, 125)
    np.testing.assert_array_equal(d.cpu().numpy()[keep], got[keep])


def test_stage_in_place_outside_the_window(cuda, oracle_mod, adv_lib):
    """The binary64 pass over single cells of a block reads the solution that
    the block's other cells have already overwritten elsewhere."""
    cfg = dict(MESHES["uniform"], degree=4, n_cells=(5, 4, 3))
    o, op = oracle_mod.Oracle(**cfg), adv_lib.AdvectionOperation(**cfg)
    rng = np.random.default_rng(10)
    scale = np.where(np.arange(60) % 5 == 2, 2.0 ** -700, 1.0)[:, None]
    u0, r0 = ((rng.standard_normal((60, 125)) * scale).reshape(-1) for _ in range(2))
    uo, ro = u0.copy(), r0.copy()
    o.perform_stage(0.0, 0.013, 0.021, ro, np.zeros_like(u0), uo, ro)
    u, r, k = cuda.from_numpy(u0).cuda(), cuda.from_numpy(r0).cuda(), op.initialize_dof_vector()
    op.perform_stage(0.0, 0.013, 0.021, r, k, u, r)
    assert np.abs(u.cpu().numpy() - uo).max() <= TOL * np.abs(uo).max()
    assert np.abs(r.cpu().numpy() - ro).max() <= TOL * np.abs(ro).max()


@pytest.mark.parametrize("degree", [1, 4, 5])
@pytest.mark.parametrize("curved", [0, 1])
def test_step_across_the_sign_change_of_the_velocity(cuda, oracle_mod, adv_lib, curved, degree):
    """cos(pi t / 0.5) changes sign at t = 0.25: the upwind side changes
    between the stage that writes a trace and the one that reads it."""
    cfg = dict(MESHES["rotating"], degree=degree, mesh_type=curved, deformation=0.05 * curved)
    u0 = np.random.default_rng(degree).standard_normal(oracle_mod.Oracle(**cfg).n_dofs)
    ref = oracle_step(oracle_mod, cfg, u0, 0.2495, 0.002)
    got = gpu_step(cuda, adv_lib, cfg, u0, 0.2495, 0.002)
    assert np.abs(got - ref).max() <= TOL * np.abs(ref).max()


def test_uniform_velocity_with_a_zero_component(cuda, oracle_mod, adv_lib):
    """No flux along y reads a trace; the binary64 path (first scale) must not
    use the ones that were never written either."""
    cfg = dict(MESHES["uniform"], degree=3, velocity=(0.7, 0.0, -0.4))
    u0 = np.random.default_rng(12).standard_normal(oracle_mod.Oracle(**cfg).n_dofs)
    ref = oracle_step(oracle_mod, cfg, u0, 0.0, 0.004)
    for exponent in (-600, 0):
        junk = cuda.full((1 << 22,), float("nan"), dtype=cuda.float64, device="cuda")  # memory the traces may get
        del junk
        cuda.cuda.empty_cache()
        got = np.ldexp(gpu_step(cuda, adv_lib, cfg, np.ldexp(u0, exponent), 0.0, 0.004), -exponent)
        assert np.abs(got - ref).max() <= TOL * np.abs(ref).max()


# ---- advection-diffusion

SIPG = {
    "sipg-rotating": dict(n_cells=(3, 2, 3), periodic=0, velocity_type=1, velocity=(1.0, 1.0, 0.3), velocity_period=0.5,
                          diffusion=1e-2, initial_condition=1, ic_params=(0.3, 0.5, 0.5, 0.2), boundary_value=0),
    "sipg-periodic": dict(n_cells=(2, 3, 4), diffusion=3e-2),
    "sipg-exact": dict(n_cells=(2, 2, 3), periodic=0, diffusion=1e-3, initial_condition=2, boundary_value=1),
}


@pytest.mark.parametrize("degree", [1, 2, 3, 4, 5, 6])
@pytest.mark.parametrize("mesh", sorted(SIPG))
def test_diffusive_step_matches_oracle(cuda, oracle_mod, adv_lib, mesh, degree):
    cfg = dict(SIPG[mesh], degree=degree)
    o = oracle_mod.Oracle(**cfg)
    u0 = np.random.default_rng(degree).standard_normal(o.n_dofs)
    dt = o.time_step(0.2)
    # the sign change of the rotating velocity falls between the stages
    ref = oracle_step(oracle_mod, cfg, u0, 0.2499, dt)
    got = gpu_step(cuda, adv_lib, cfg, u0, 0.2499, dt)
    assert np.abs(got - ref).max() <= TOL * np.abs(ref).max()
    np.testing.assert_array_equal(
        got, gpu_step(cuda, adv_lib, cfg, u0, 0.2499, dt, fused_form=adv_lib.FORM_COLLOCATION_NO_TRACES))


@pytest.mark.parametrize("exponent", [-900, -300, 300, 900])
def test_diffusive_step_commutes_with_powers_of_two(cuda, oracle_mod, adv_lib, exponent):
    cfg = dict(SIPG["sipg-rotating"], degree=4)
    o = oracle_mod.Oracle(**cfg)
    u0 = np.random.default_rng(3).standard_normal(o.n_dofs)
    dt = o.time_step(0.2)
    ref = oracle_step(oracle_mod, cfg, u0, 0.0, dt)
    got = np.ldexp(gpu_step(cuda, adv_lib, cfg, np.ldexp(u0, exponent), 0.0, dt), -exponent)
    assert np.abs(got - ref).max() <= TOL * np.abs(ref).max()


@pytest.mark.parametrize("velocity, diffusion", [((0.0, 0.0, 0.0), 1e-2), ((1e-9, 0.0, 0.0), 1.0), ((1.0, 2.0, 0.0), 1e-12)])
def test_diffusive_step_scales_of_the_terms(cuda, oracle_mod, adv_lib, velocity, diffusion):
    """Pure diffusion, negligible advection, negligible diffusion."""
    cfg = dict(degree=4, n_cells=(3, 3, 2), velocity=velocity, diffusion=diffusion)
    u0 = np.random.default_rng(4).standard_normal(oracle_mod.Oracle(**cfg).n_dofs)
    dt = 1e-5
    ref = oracle_step(oracle_mod, cfg, u0, 0.0, dt)
    got = gpu_step(cuda, adv_lib, cfg, u0, 0.0, dt)
    assert np.abs(got - ref).max() <= TOL * np.abs(ref).max()
