"""Scale of the block fixed-point SIPG stage: the increment (u_new - u_0) / dt
against the oracle where diffusion is the only term that counts, so that a
unit set by a velocity that is not there (or is multiplied by zero) shows.

Bar: 1e-12 of the increment's largest entry.  At dt a twentieth of h^2 / (nu n^4)
the increment is a few per cent of u, whose rounding (2^-53) is then some
1e-14 of it.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = 1e-12


def increments(torch, oracle_mod, adv, cfg, t, dt, seed):
    o, op = oracle_mod.Oracle(**cfg), adv.AdvectionOperation(**cfg)
    u0 = np.random.default_rng(seed).standard_normal(o.n_dofs)
    ref = u0.copy()
    o.lsrk_step(t, dt, ref, np.zeros_like(u0), np.zeros_like(u0))
    u, r, k = torch.from_numpy(u0).cuda(), op.initialize_dof_vector(), op.initialize_dof_vector()
    op.lsrk_steps(adv.LSRK_5_4, t, dt, 1, u, r, k)
    return (u.cpu().numpy() - u0) / dt, (ref - u0) / dt


def diffusive_step(cfg, edge):
    return 0.05 * (edge / max(cfg["n_cells"])) ** 2 / (cfg["diffusion"] * (cfg["degree"] + 1) ** 4)


@pytest.mark.parametrize("degree", [1, 3, 6])
@pytest.mark.parametrize("edge", [1.0, 1e-3])
@pytest.mark.parametrize("nu", [1e-3, 1e-6, 1e-9, 1e-16])
def test_diffusion_without_velocity(cuda, oracle_mod, adv_lib, nu, edge, degree):
    cfg = dict(degree=degree, n_cells=(3, 3, 2), velocity=(0.0, 0.0, 0.0), diffusion=nu, domain_hi=(edge,) * 3)
    got, ref = increments(cuda, oracle_mod, adv_lib, cfg, 0.0, diffusive_step(cfg, edge), degree)
    assert np.abs(ref).max() > 0.0
    assert np.abs(got - ref).max() <= TOL * np.abs(ref).max()


@pytest.mark.parametrize("degree", [1, 3, 6])
@pytest.mark.parametrize("nu", [1e-3, 1e-9])
def test_diffusion_while_the_velocity_reverses(cuda, oracle_mod, adv_lib, nu, degree):
    """cos(pi t / T) is 6e-17 at t = T / 2; T is so long that dt does not move t."""
    period = 1e25
    cfg = dict(degree=degree, n_cells=(3, 2, 3), periodic=0, velocity_type=1, velocity=(1.0, 1.0, 0.3),
               velocity_period=period, diffusion=nu, initial_condition=1, ic_params=(0.3, 0.5, 0.5, 0.2),
               boundary_value=0)
    dt = diffusive_step(cfg, 1.0)
    assert period / 2 + dt == period / 2
    got, ref = increments(cuda, oracle_mod, adv_lib, cfg, period / 2, dt, degree)
    assert np.abs(got - ref).max() <= TOL * np.abs(ref).max()
