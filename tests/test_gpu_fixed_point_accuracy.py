"""Accuracy of the block fixed-point operator against extended precision.

The operator of a periodic cube in the library's own discretization, built
here in numpy's extended precision (64 bits of mantissa or more), gives the
errors of the fixed-point kernels.  They are compared with those of the
library's binary64 kernels on the same data: with the velocity 2^250 times
as large the metric lies outside the fixed-point window, and every result
of those kernels is 2^250 times that of the original velocity, bit for bit.

Bars, on the error's norm averaged over six seeds: apply at most 1.15 times
binary64's (0.73 to 1.09 measured; one bit less in the scale of U gives 1.32
for degree 5) and at most the oracle's (0.42 to 0.97); a step at most 1.05
times binary64's stages (0.99 to 1.01; both change bases in fixed point) and
8 * 2^-53 of the result (2.5 to 5.8).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

X = np.longdouble
VELOCITY = (1.0, 0.15, -0.05)
CELLS = (2, 3, 2)


def legendre(n, x):
    p, q = np.ones_like(x), x
    for k in range(2, n + 1):
        p, q = q, ((2 * k - 1) * x * q - (k - 1) * p) / k
    return q, n * (x * q - p) / (x * x - 1)


def gauss(n):
    x = np.polynomial.legendre.leggauss(n)[0].astype(X)
    for _ in range(6):
        p, d = legendre(n, x)
        x = x - p / d
    d = legendre(n, x)[1]
    return (1 + x) / 2, 1 / ((1 - x * x) * d * d)


def lobatto(n):
    m = n - 1
    x = np.sort(np.polynomial.legendre.Legendre.basis(m).deriv().roots().real).astype(X)
    for _ in range(6):
        p, d = legendre(m, x)
        x = x - d * (1 - x * x) / (2 * x * d - m * (m + 1) * p)
    return np.concatenate([[X(0)], (1 + x) / 2, [X(1)]])


def lagrange(nodes, x):
    """Values and derivatives of the Lagrange polynomials at x, [point, polynomial]."""
    n, x = len(nodes), np.asarray(x, X)

    def product(i, skip=()):
        f = np.ones_like(x)
        for j in range(n):
            if j != i and j not in skip:
                f = f * (x - nodes[j]) / (nodes[i] - nodes[j])
        return f

    d = [sum(product(i, (m,)) / (nodes[i] - nodes[m]) for m in range(n) if m != i) for i in range(n)]
    return np.stack([product(i) for i in range(n)], 1), np.stack(d, 1)


class Operator:
    """-div(a u) with upwind fluxes on the unit cube, degree n - 1."""

    def __init__(self, n):
        self.n = n
        gp, gw = gauss(n)
        self.S = lagrange(lobatto(n), gp)[0]
        self.Si = lagrange(gp, lobatto(n))[0]
        self.Dw = lagrange(gp, gp)[1].T * gw[None, :] / gw[:, None]
        self.l = lagrange(gp, [0, 1])[0]
        self.lift = self.l / gw

    def along(self, m, u, d):
        return np.moveaxis(np.tensordot(m, u, axes=([1], [5 - d])), 0, 5 - d)

    def sweep(self, m, u):
        for d in range(3):
            u = self.along(m, u, d)
        return u

    def rate(self, u):
        z = 0
        for d in range(3):
            c = X(VELOCITY[d]) * CELLS[d]
            out = self.along(self.l[1 if c > 0 else 0][None], u, d)
            inflow = np.roll(out, 1 if c > 0 else -1, 2 - d)
            low, high = (inflow, out) if c > 0 else (out, inflow)
            z = z + c * (self.along(self.Dw, u, d) + self.along(self.lift[0][:, None], low, d)
                         - self.along(self.lift[1][:, None], high, d))
        return z

    def to_gauss(self, u):
        return self.sweep(self.S, np.asarray(u, X).reshape(CELLS[::-1] + (self.n,) * 3))

    def apply(self, u):
        return self.sweep(self.Si, self.rate(self.to_gauss(u))).reshape(-1)

    def step(self, u, dt, a, b):
        u = self.to_gauss(u)
        r = u
        for i in range(len(b)):
            k = self.rate(r)
            if i < len(b) - 1:
                r = u + X(a[i]) * X(dt) * k
            u = u + X(b[i]) * X(dt) * k
        return self.sweep(self.Si, u).reshape(-1)


def size(x):
    return float(np.sqrt((x * x).sum()))


@pytest.mark.parametrize("degree", [1, 2, 3, 4, 5, 6])
@pytest.mark.parametrize("data", ["random", "20 binades"])
def test_errors_against_extended_precision(cuda, oracle_mod, adv_lib, data, degree):
    exact = Operator(degree + 1)
    dt, (a, b) = 2.0 ** -9, adv_lib.lsrk_coefficients(adv_lib.LSRK_3_3)
    o = oracle_mod.Oracle(degree=degree, n_cells=CELLS, velocity=VELOCITY)
    scales = (1.0, 2.0 ** 250)  # fixed point, binary64
    ops = [adv_lib.AdvectionOperation(degree=degree, n_cells=CELLS, velocity=tuple(s * v for v in VELOCITY))
           for s in scales]
    applied, stepped, by_oracle = np.zeros(2), np.zeros(2), 0.0
    for seed in range(6):
        rng = np.random.default_rng(seed)
        u = rng.standard_normal(o.n_dofs)
        if data != "random":
            u *= np.exp2(rng.uniform(-20, 0, o.n_dofs))
        ea, es = exact.apply(u), exact.step(u, dt, a, b)
        by_oracle += size(o.apply(u, 0.0) - ea) / size(ea) / 6
        for i, (op, s) in enumerate(zip(ops, scales)):
            v, r, k = cuda.from_numpy(u).cuda(), op.initialize_dof_vector(), op.initialize_dof_vector()
            op.apply(v, r, 0.0)
            applied[i] += size(r.cpu().numpy().astype(X) / X(s) - ea) / size(ea) / 6
            op.lsrk_steps(adv_lib.LSRK_3_3, 0.0, dt / s, 1, v, r, k)
            stepped[i] += size(v.cpu().numpy() - es) / size(es) / 6
    assert applied[0] <= 1.15 * applied[1] and applied[0] <= by_oracle
    assert stepped[0] <= 1.05 * stepped[1] and stepped[0] <= 8 * 2.0 ** -53
