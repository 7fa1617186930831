"""The radial line operators where their paths change, in every configuration,
against the oracle: one row per thread or two (T and T + 1 points), last
threads with and without rows, lines that end around the 64 (derivatives) and
128 rows (filter) whose factors a block keeps, and around the rows from which
the factors are constants (15, 23 and 90) with the four end rows behind.  The
bound is the one of the other operator tests, 1e-12 of each line's maximum."""
import numpy as np
import pytest

from conftest import rel_err

pytestmark = pytest.mark.gpu
SHORT_T, LONG_T = (64, 128, 256), (256, 512, 1024)


def lengths(cfg):
    t, u = SHORT_T[cfg], LONG_T[cfg]
    n = {16, 17, 18, 19, 20, 26, 27, 28, 66, 67, 68, 69, 70, 93, 94, 95, 96, 130, 131, 132, 133, 134, 1023, 1024}
    n |= {m for k in range(1, 5) for m in (k * t - 1, k * t, k * t + 1)} | {t + t // 2, 4 * t - 5}
    n |= {m for k in range(1, 17) for m in (k * u - 1, k * u, k * u + 1) if k in (1, 2, 3, 4, 16)} | {2 * u + 7, 4 * u - 5}
    return sorted(m for m in n if 16 <= m <= 4096)


@pytest.mark.parametrize("cfg", [0, 1, 2])
def test_line_operators(oracle_mod, cfg):
    from shock_turbulence_b200.params import radial_params
    from shock_turbulence_b200.radial import RadialBatch
    ns = np.asarray(lengths(cfg), dtype=np.int32)
    b = RadialBatch(ns, np.full(len(ns), 2.0))
    b.config(cfg, cfg)
    o = oracle_mod.Radial(radial_params())
    rng = np.random.default_rng(cfg)
    F = rng.standard_normal(b.npts)
    d, d2, e, f, g = (rng.standard_normal(b.npts) for _ in range(5))
    r = [x.copy() for x in (d, d2, e, f, g)]
    b.DFDX(F, d, 1, -0.5)
    b.D2FDX2(F, e, d2, 1)
    b.Compact_Filter_X(F, f)
    b.Gaussian_Filter_X(F, g)
    off = 0
    for n in ns:
        s = slice(off, off + n)
        o.dfdx(2.0, F[s], r[0][s], 1, -0.5)
        o.d2fdx2(2.0, F[s], r[2][s], r[1][s], 1)
        o.filter(F[s], r[3][s])
        o.gauss(F[s], r[4][s])
        for what, x, y in zip(("DFDX", "D2FDX2", "its DFDX", "filter", "Gauss"), (d, d2, e, f, g), r):
            assert rel_err(x[s], y[s]) < 1e-12, (what, n)
        off += n
    b.close()
