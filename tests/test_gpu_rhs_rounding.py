"""RHS adds the derivative of the momentum flux and that of the pressure (the
reference's two calls), it does not differentiate their sum: with one velocity
component and no viscosity, the momentum right-hand side of that component has
the bits of the reference's expressions evaluated with the single operators."""
import numpy as np
import pytest

from shock_turbulence_b200.params import default_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("grid", [(48, 32, 64), (112, 48, 16), (16, 112, 48)])
@pytest.mark.parametrize("d", [0, 1, 2])
def test_momentum_bits(d, grid):
    from shock_turbulence_b200 import Solver
    s = Solver(default_params(*grid))
    rng = np.random.default_rng(d)
    q, rho = 0.3 * rng.standard_normal(s.shape), rng.uniform(0.8, 1.2, s.shape)
    E, Y = rng.uniform(2.0, 3.0, s.shape), np.ones(s.shape)
    Q = np.zeros((5,) + s.shape)
    Q[d], Q[3], Q[4] = q, rho, E
    s.Compute_gamma(Y)
    g = s.get_common("gamma_eff")
    Vs = 1.0 / rho
    u, P = q * Vs, (g - 1.0) * (E - 0.5 * Vs * (q * q))
    name = "DFD" + "XYZ"[d]
    sym, asym = getattr(s, name + "_sym"), getattr(s, name + "_asym")
    f, fr, du = s.field(), s.field(), s.field()
    sym(q * u, f, 0, -0.5)
    sym(P, f, 1, -1.0)
    asym(q, fr, 0, 1.0)
    asym(u, du, 0, 1.0)
    want = (f + (-0.5 * fr) * u) + (-0.5 * rho * u) * du
    rhs = s.field(5)
    s.RHS(Q, rhs, Y)
    assert np.array_equal(rhs[d], want)


def test_viscosity_slope_is_a_power():
    """The heat flux of a fluid at rest: Pri (mu d2T + dmu/dT (dT)^2), with the
    bits that powers rounded to nearest give.  Where the slope's term is five
    times the other, CPU powers (0.52 ulp) give them on 97 % of the cells, a
    quotient in place of the slope's power on 81 %; CUDA's power is off by one
    ulp on few cells, so 0.9 tells the two apart."""
    from shock_turbulence_b200 import Solver
    nx, ny, nz = 512, 16, 16
    p = default_params(nx, ny, nz, re=100.0)
    s = Solver(p)
    x = np.arange(nx) * (p.x_leng / (nx - 1))
    rho = np.broadcast_to((0.4 / (1.75 + 1.2 * np.cos(x)))[:, None, None], s.shape).copy()
    E, Y = np.full(s.shape, 2.5), np.ones(s.shape)
    Q = np.zeros((5,) + s.shape)
    Q[3], Q[4] = rho, E
    s.Compute_gamma(Y)
    g = s.get_common("gamma_eff")
    fac1, fac3 = p.gamma1 - 1.0, p.gamma1 / (p.gamma1 - 1.0)
    T = fac3 * (1.0 / rho) * ((g - 1.0) * E)
    d1, d2 = [s.field() for _ in range(3)], [s.field() for _ in range(3)]
    for k, c in enumerate("XYZ"):
        getattr(s, f"D2FD{c}2_sym")(T, d1[k], d2[k], 1)
    L = np.longdouble
    X = (fac1 * T).astype(L)
    Re_inv, Pri = 1.0 / p.re1, 1.0 / p.pr
    mu = (X ** L(p.vis_exp)).astype(np.float64) * Re_inv
    dmu = (X ** L(p.vis_exp - 1.0)).astype(np.float64) * Re_inv * p.vis_exp * fac1
    want = Pri * (mu * d2[0] + dmu * d1[0] * d1[0]) + Pri * (mu * (d2[1] + d2[2]) + dmu * (d1[1] * d1[1] + d1[2] * d1[2]))
    rhs = s.field(5)
    s.RHS(Q, rhs, Y)
    k = np.abs(mu * d2[0]) < 0.2 * dmu * d1[0] * d1[0]
    assert k.mean() > 0.05
    assert (rhs[4] == want)[k].mean() > 0.9
