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
