"""Block fixed-point kernels near the lower end of the binary64 range."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = 1e-12

MESHES = {
    "uniform": dict(n_cells=(3, 2, 5)),
    "curved": dict(n_cells=(3, 3, 2), mesh_type=1, deformation=0.07),
    "sipg": dict(n_cells=(3, 2, 3), diffusion=3e-2),
}


def gpu_step(torch, adv, cfg, u0, dt, **kw):
    op = adv.AdvectionOperation(**cfg, **kw)
    u, r, k = torch.from_numpy(np.ascontiguousarray(u0)).cuda(), op.initialize_dof_vector(), op.initialize_dof_vector()
    op.lsrk_steps(adv.LSRK_5_4, 0.0, dt, 1, u, r, k)
    return u.cpu().numpy()


def oracle_step(o, u0, dt):
    u = u0.copy()
    o.lsrk_step(0.0, dt, u, np.zeros_like(u0), np.zeros_like(u0))
    return u


@pytest.mark.parametrize("mesh", sorted(MESHES))
def test_values_below_the_normal_range(cuda, oracle_mod, adv_lib, mesh):
    """Data near 2^-1050, whose high words are zero, among cells of zeros.

    The quantum is 2^-1074.  A step's sums and changes of basis amplify their
    roundings to some 2^12 quanta of a result of 2^25; apply multiplies them
    by 1 / det J <= 45 and S^-1, some 2^18 quanta of a result of 2^30.
    """
    cfg = dict(MESHES[mesh], degree=3)
    o = oracle_mod.Oracle(**cfg)
    u0 = np.ldexp(np.random.default_rng(1).standard_normal(o.n_dofs), -1050).reshape(-1, 64)
    u0[::3] = 0.0
    u0 = u0.reshape(-1)
    assert np.abs(u0).max() < 2.0 ** -1042
    dt = 1e-3
    ref = oracle_step(o, u0, dt)
    for form in (adv_lib.FORM_AUTO, adv_lib.FORM_COLLOCATION_NO_TRACES):
        got = gpu_step(cuda, adv_lib, cfg, u0, dt, fused_form=form)
        assert np.abs(got - ref).max() <= 2.0 ** -10 * np.abs(ref).max()
    op = adv_lib.AdvectionOperation(**cfg)
    s, d = cuda.from_numpy(u0).cuda(), op.initialize_dof_vector()
    op.apply(s, d, 0.0)
    ref = o.apply(u0, 0.0)
    assert np.abs(d.cpu().numpy() - ref).max() <= 2.0 ** -9 * np.abs(ref).max()


@pytest.mark.parametrize("exponent", [-760, -740, -720, -700, -560, -410, -395])
@pytest.mark.parametrize("mesh", sorted(MESHES))
def test_blocks_near_the_lower_end_of_the_window(cuda, oracle_mod, adv_lib, mesh, exponent):
    """Cells of 2^(exponent + 0..24): some blocks inside, some outside the window."""
    cfg = dict(MESHES[mesh], degree=3)
    o, op = oracle_mod.Oracle(**cfg), adv_lib.AdvectionOperation(**cfg)
    rng = np.random.default_rng(2)
    u0 = (rng.standard_normal((o.n_dofs // 64, 64)) * np.exp2(rng.integers(0, 25, (o.n_dofs // 64, 1)))).reshape(-1)
    got = np.ldexp(gpu_step(cuda, adv_lib, cfg, np.ldexp(u0, exponent), 1e-3), -exponent)
    ref = oracle_step(o, u0, 1e-3)
    assert np.abs(got - ref).max() <= TOL * np.abs(ref).max()
    s, d = cuda.from_numpy(np.ldexp(u0, exponent)).cuda(), op.initialize_dof_vector()
    op.apply(s, d, 0.0)
    ref = o.apply(u0, 0.0)
    assert np.abs(np.ldexp(d.cpu().numpy(), -exponent) - ref).max() <= TOL * np.abs(ref).max()


@pytest.mark.parametrize("mesh", ["uniform", "curved"])
def test_small_cells_keep_their_own_accuracy(cuda, oracle_mod, adv_lib, mesh):
    """Cells of 2^-470 that no value of 1 reaches within the step's five stages."""
    cfg = dict(MESHES[mesh], degree=4, n_cells=(16, 2, 2))
    o = oracle_mod.Oracle(**cfg)
    u0 = np.random.default_rng(5).standard_normal((4, 16, 125))
    u0[:, 1:] *= 2.0 ** -470
    u0 = u0.reshape(-1)
    ref, got = oracle_step(o, u0, 1e-3).reshape(-1, 125), gpu_step(cuda, adv_lib, cfg, u0, 1e-3).reshape(-1, 125)
    size = np.abs(ref).max(axis=1)
    small = size < 2.0 ** -400
    assert small.sum() >= 4 * 5
    assert (np.abs(got - ref).max(axis=1) <= TOL * size)[small].all()
