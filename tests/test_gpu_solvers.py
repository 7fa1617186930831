"""The general line solvers at the ends of their ranges, against the oracle:
the shortest lines of each elimination, row counts around the sweeps' blocks
(8, 6 and 4 rows, double-buffered), line counts around a warp, coefficients
and right-hand sides on the host, on the device and overlapping.  Kernels and
oracle do the same operations in the same order; 1e-14 leaves room for the
conditioning (diagonally dominant rows)."""
import numpy as np
import pytest

from conftest import rel_err
from shock_turbulence_b200.params import default_params

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def solver():
    from shock_turbulence_b200 import Solver
    s = Solver(default_params(16))
    yield s
    s.close()


def rows(rng, n, lot, *mids):
    return [m + 0.05 * rng.standard_normal((n, lot)) for m in mids]


@pytest.mark.parametrize("lot", [1, 31, 33, 200])
@pytest.mark.parametrize("n", [1, 2, 3, 4, 7, 8, 9, 12, 13, 17, 33, 100])
@pytest.mark.parametrize("nper", [0, 1])
def test_tridiagonal(solver, oracle_mod, n, lot, nper):
    import torch
    rng = np.random.default_rng(n * 1000 + lot)
    A, B, C, R = rows(rng, n, lot, 0.3, 1.0, 0.3, 0.0)
    r = R.copy()
    oracle_mod.tridiagonal(A.copy(), B.copy(), C.copy(), r, nper)
    host = R.copy()
    solver.tridiagonal(A, B, C, host, n, lot, nper)
    assert rel_err(host, r) < 1e-14
    dev = [torch.from_numpy(x).cuda() for x in (A, B, C, R)]
    torch.cuda.synchronize()
    solver.tridiagonal(*dev, n, lot, nper)
    assert np.array_equal(dev[3].cpu().numpy(), host)
    assert all(np.array_equal(d.cpu().numpy(), x) for d, x in zip(dev, (A, B, C)))


@pytest.mark.parametrize("lot", [1, 33, 200])
@pytest.mark.parametrize("n", [1, 2, 3, 4, 5, 6, 7, 8, 9, 12, 13, 17, 33, 100])
@pytest.mark.parametrize("nper", [0, 1])
def test_pentadiagonal(solver, oracle_mod, n, lot, nper):
    import torch
    from shock_turbulence_b200 import StError
    rng = np.random.default_rng(n * 1000 + lot)
    co = rows(rng, n, lot, 0.05, 0.25, 1.0, 0.25, 0.05)
    R = rng.standard_normal((n, lot))
    host = R.copy()
    if nper and n < 5:
        with pytest.raises(StError):
            solver.pentadiagonal(*co, host, n, lot, nper)
        return
    r = R.copy()
    oracle_mod.pentadiagonal(*(x.copy() for x in co), r, nper)
    solver.pentadiagonal(*co, host, n, lot, nper)
    assert rel_err(host, r) < 1e-14
    dev = [torch.from_numpy(x).cuda() for x in (*co, R)]
    torch.cuda.synchronize()
    solver.pentadiagonal(*dev, n, lot, nper)
    assert np.array_equal(dev[5].cpu().numpy(), host)


@pytest.mark.parametrize("nper", [0, 1])
def test_overlapping_right_hand_side(solver, nper):
    """R in the array of a coefficient that the back substitution still reads."""
    import torch
    n, lot = 20, 40
    rng = np.random.default_rng(3)
    A, B, C = (torch.from_numpy(x).cuda() for x in rows(rng, n, lot, 0.3, 1.0, 0.3))
    x = C.clone()
    torch.cuda.synchronize()
    solver.tridiagonal(A, B, C.clone(), x, n, lot, nper)
    y = C.clone()
    torch.cuda.synchronize()
    solver.tridiagonal(A, B, y, y, n, lot, nper)
    assert torch.equal(x, y)


def test_memory_counts_the_workspace():
    """st_memory follows the solvers' workspace: room for one field of a
    tridiagonal solve of device arrays, for its four arrays too from the host."""
    import ctypes
    import torch
    from shock_turbulence_b200 import Solver

    def held(s):
        b = ctypes.c_longlong()
        assert s.lib.st_memory(s._h, ctypes.byref(b)) == 0
        return b.value

    s = Solver(default_params(16))
    n, lot = 100, 200
    rng = np.random.default_rng(4)
    host = rows(rng, n, lot, 0.3, 1.0, 0.3, 0.0)
    dev = [torch.from_numpy(x).cuda() for x in host]
    torch.cuda.synchronize()
    start = held(s)
    s.tridiagonal(*dev, n, lot, 0)
    assert held(s) - start == 8 * n * lot
    s.tridiagonal(*host, n, lot, 0)
    assert held(s) - start == 5 * 8 * n * lot
    s.close()


def test_workspace_makes_room_for_scratch():
    """On a device that is full but for 32 MiB, a routine whose scratch fields
    need more gets the room that a large solve has left in its context."""
    import torch
    from shock_turbulence_b200 import Solver
    p = default_params(64, 64, 64, re=100.0)
    s, other = Solver(p), Solver(p)
    rng = np.random.default_rng(8)
    Q = np.empty((5,) + s.shape)
    Q[:3], Q[3], Q[4] = 0.1 * rng.standard_normal((3,) + s.shape), 1.0, 2.0
    Y = np.full(s.shape, 0.5)
    ref = other.field(5)
    other.Compute_gamma(Y)
    other.RHS(Q.copy(), ref, Y)
    other.close()
    n, lot = 512, 120000                       # half a gigabyte of workspace
    co = [torch.full((n * lot,), v, dtype=torch.float64, device="cuda") for v in (0.3, 1.0, 0.3, 0.0)]
    torch.cuda.synchronize()
    s.tridiagonal(*co, n, lot, 0)
    del co
    torch.cuda.empty_cache()
    full = []
    for size in (1 << 30, 1 << 25, 1 << 21):
        while torch.cuda.mem_get_info()[0] > size + (1 << 25):
            try:
                full.append(torch.empty(size, dtype=torch.uint8, device="cuda"))
            except torch.OutOfMemoryError:
                break
    out = s.field(5)
    try:
        s.Compute_gamma(Y)
        s.RHS(Q.copy(), out, Y)
    finally:
        del full
        torch.cuda.empty_cache()
        s.close()
    assert np.array_equal(out, ref)
