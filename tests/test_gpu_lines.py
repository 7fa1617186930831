"""The line kernel at the edges of its dispatch, against the oracle.

A line of n rows is cut into segments of 8 (n < 96) or 16 rows, at most 32;
tiles hold 16 columns, or 8 where four tiles of a launch do not fit (lines of
more than about 430 rows); x and z tiles of more than 256 rows move in two
transfers; the number of slots and CTAs follows from the tile size.  Each
direction takes the smallest line (16), both sides of every switch and the
largest (512).  The operators are held to 1e-12 and whole steps (every pair
and product that the right-hand sides form) to 1e-10, the bounds that the
other parity tests use; the FP32 mode's step to 1e-5 of the FP64 one."""
import numpy as np
import pytest

from conftest import rel_err
from shock_turbulence_b200.params import PRECISION_FP32, default_params, periodic_params

pytestmark = pytest.mark.gpu
DIRS = "XYZ"
GRIDS = [(512, 16, 16), (16, 512, 16), (16, 16, 512), (448, 32, 16), (16, 448, 32), (32, 16, 448), (80, 96, 256),
         (272, 80, 96), (96, 272, 80)]


def octant(grid, **kw):
    """Uniform spacing: the artificial viscosity scales with the x spacing."""
    nx, ny, nz = grid
    return default_params(nx, ny, nz, re=100.0, c_beta_scale=1.75, x_leng=(nx - 1) / 64.0, y_leng=(ny - 1) / 64.0,
                          z_leng=(nz - 1) / 64.0, **kw)


def blast(p, seed=7):
    from shock_turbulence_b200.initial import blast_in_turbulence
    return blast_in_turbulence(p, k0=2, mach_t=0.1, p_ratio=20.0, radius_cells=4, seed=seed)


def one_step(h, Q, Y):
    """Set-up and one main-loop step of a Solver or an Oracle."""
    h.set_state(Q, Y)
    for name, args in (("Compute_gamma", (Y,)), ("Compute_hyper", (Q, Y))):
        getattr(h, name if hasattr(h, name) else name.lower())(*args)
    h.step(0.0, 0)
    return h.get_state()


@pytest.mark.parametrize("grid", GRIDS)
@pytest.mark.parametrize("family", ["octant", "periodic"])
def test_operators(oracle_mod, grid, family):
    from shock_turbulence_b200 import Solver
    p = default_params(*grid, length=2.0, re=100.0) if family == "octant" else periodic_params(*grid)
    s, o = Solver(p), oracle_mod.Oracle(p)
    rng = np.random.default_rng(sum(grid))
    for d in range(3):
        for asym in ((0, 1) if family == "octant" else (0,)):
            sfx = "" if family == "periodic" else ("_asym" if asym else "_sym")
            F, g = rng.standard_normal(s.shape), rng.standard_normal(s.shape)
            r = g.copy()
            getattr(s, f"DFD{DIRS[d]}{sfx}")(F, g, 1, -0.5)
            o.dfd(d, asym, F, r, 1, -0.5)
            assert rel_err(g, r) < 1e-12, ("DFD", d, asym)
            g1, g2, r1, r2 = (np.zeros(s.shape) for _ in range(4))
            getattr(s, f"D2FD{DIRS[d]}2{sfx}")(F, g1, g2, 1)
            o.d2fd2(d, asym, F, r1, r2, 1)
            assert rel_err(g2, r2) < 1e-12 and rel_err(g1, r1) < 1e-12, ("D2FD2", d, asym)
            getattr(s, f"D2FD{DIRS[d]}2{sfx}")(F, None, g2, 0)
            assert rel_err(g2, r2) < 1e-12, ("D2FD2 alone", d, asym)
            getattr(s, f"Compact_Filter_{DIRS[d]}{sfx}")(F, g)
            o.filter(d, asym, F, r)
            assert rel_err(g, r) < 1e-12, ("filter", d, asym)
    s.close()


@pytest.mark.parametrize("grid", GRIDS)
def test_whole_step(oracle_mod, grid):
    from shock_turbulence_b200 import Solver
    p = octant(grid)
    Q, Y = blast(p)
    s = Solver(p)
    Qg, Yg = one_step(s, Q, Y)
    s.close()
    Qo, Yo = one_step(oracle_mod.Oracle(p), Q, Y)
    for l in range(5):
        assert rel_err(Qg[l], Qo[l]) < 1e-10, l
    assert rel_err(Yg, Yo) < 1e-10


@pytest.mark.parametrize("grid", [(448, 32, 16), (16, 448, 32), (32, 32, 448), (80, 96, 272)])
def test_fp32_step(grid):
    from shock_turbulence_b200 import Solver
    out = []
    for prec in (0, PRECISION_FP32):
        p = octant(grid, precision=prec)
        Q, Y = blast(p)
        s = Solver(p)
        out.append(one_step(s, Q, Y))
        s.close()
    for l in range(5):
        assert rel_err(out[1][0][l], out[0][0][l]) < 1e-5, l
    assert rel_err(out[1][1], out[0][1]) < 1e-5


def test_unaligned_fields():
    """Device fields that start 8 bytes off a 16-byte boundary give the same
    bits as aligned ones, in place too."""
    import torch
    from shock_turbulence_b200 import Solver
    s = Solver(default_params(32, 48, 16, length=2.0))
    n = s.n3
    F = torch.randn(n, dtype=torch.float64, device="cuda", generator=torch.Generator("cuda").manual_seed(1))

    def off(x):
        b = torch.empty(n + 1, dtype=torch.float64, device="cuda")
        b[1:] = x
        return b[1:]
    for d in DIRS:
        a, b, G = torch.ones_like(F), off(torch.ones_like(F)), off(F)
        torch.cuda.synchronize()
        getattr(s, f"DFD{d}_sym")(F, a, 1, -0.5)
        getattr(s, f"DFD{d}_sym")(G, b, 1, -0.5)
        assert torch.equal(a, b)
        getattr(s, f"Compact_Filter_{d}_asym")(F, a)
        getattr(s, f"Compact_Filter_{d}_asym")(G, G)
        assert torch.equal(a, G)
    s.close()


@pytest.mark.parametrize("n", [16, 64, 112, 400, 512])
@pytest.mark.parametrize("d", [0, 1, 2])
def test_derivatives_in_place(d, n):
    """An output that is the operand's array: the bits of separate arrays (each
    tile is read before it is written, whatever the number of slots)."""
    import torch
    from shock_turbulence_b200 import Solver
    grid = [32, 32, 32]
    grid[d] = n
    s = Solver(default_params(*grid))
    F = torch.from_numpy(np.random.default_rng(n).standard_normal(s.shape)).cuda()
    d1, d2 = getattr(s, f"DFD{DIRS[d]}_asym"), getattr(s, f"D2FD{DIRS[d]}2_sym")

    def run(op, x, *rest):
        torch.cuda.synchronize()
        op(x, *rest)

    for iadd in (0, 1):
        own, same = F.clone(), F.clone()
        run(d1, F, own, iadd, 0.7)
        run(d1, same, same, iadd, 0.7)
        assert torch.equal(own, same), iadd
    a, a2, b2 = torch.zeros_like(F), torch.zeros_like(F), torch.zeros_like(F)
    run(d2, F, a, a2, 1)
    b = F.clone()
    run(d2, b, b, b2, 1)
    assert torch.equal(a, b) and torch.equal(a2, b2)
    b, b1 = F.clone(), torch.zeros_like(F)
    run(d2, b, b1, b, 1)
    assert torch.equal(a, b1) and torch.equal(a2, b)
