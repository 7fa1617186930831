"""The outflow faces of bc_RHS, whose pressure derivative is eliminated over at
most the last 48 rows of a line: lines shorter than that, exactly as long and
longer, in each direction, against the oracle.  1e-10 of each face's largest
value, as for the other routines that compound line solves; the rows left out
weigh 2e-20."""
import numpy as np
import pytest

from conftest import rel_err
from test_gpu_lines import blast, octant

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("grid", [(16, 48, 64), (64, 16, 48), (48, 64, 16), (32, 32, 32), (80, 112, 96)])
def test_faces(oracle_mod, grid):
    from shock_turbulence_b200 import Solver
    p = octant(grid)
    Q, Y = blast(p)
    out = []
    for h, rhs, gamma, bc in ((Solver(p), "RHS", "Compute_gamma", "bc_RHS"),
                              (oracle_mod.Oracle(p), "rhs", "compute_gamma", "bc_rhs")):
        h.set_state(Q, Y)
        getattr(h, gamma)(Y)
        q, r, yr = Q.copy(), np.zeros_like(Q), np.zeros_like(Y)
        getattr(h, rhs)(q, r, Y)
        getattr(h, bc)(q, r, Y, yr)
        out.append((q, r, yr))
    (qg, rg, yg), (qo, ro, yo) = out
    assert np.array_equal(qg, qo)
    for l in range(5):
        for face in (np.s_[-1, :, :], np.s_[:, -1, :], np.s_[:, :, -1]):
            assert np.isfinite(ro[l][face]).all()
            assert rel_err(rg[l][face], ro[l][face]) < 1e-10, (l, face)
    assert rel_err(yg, yo) < 1e-10
