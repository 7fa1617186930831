"""st_step replays a captured graph from its third step on grids of up to 128^3:
the bits of steps that are launched one by one (as they are while profiling),
also when the stream changes between replays."""
import ctypes

import numpy as np
import pytest

from shock_turbulence_b200.params import PRECISION_FP32, default_params, periodic_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [0, PRECISION_FP32])
@pytest.mark.parametrize("family", ["octant", "periodic"])
def test_replayed_steps_are_launched_steps(family, precision):
    import torch
    from shock_turbulence_b200 import Solver
    from shock_turbulence_b200.initial import blast_in_turbulence
    octant = default_params(48, 32, 64, re=100.0, c_beta_scale=1.75, precision=precision)
    Q, Y = blast_in_turbulence(octant, k0=2, mach_t=0.1, p_ratio=20.0 if family == "octant" else 1.0, radius_cells=4, seed=3)
    p = octant if family == "octant" else periodic_params(48, 32, 64, precision=precision)
    other = torch.cuda.Stream()

    def run(profile, streams):
        s = Solver(p)
        Yk = Y if family == "octant" else None
        s.set_state(Q, Yk)
        if family == "octant":
            s.Compute_gamma(Y)
        s.Compute_hyper(Q, Yk)
        assert s.lib.st_profile(s._h, int(profile)) == 0
        t, k = 0.0, 0
        for i in range(6):
            assert s.lib.st_set_stream(s._h, ctypes.c_void_p(streams[i % len(streams)])) == 0
            t, k = s.step(t, k)
        out = s.get_state()
        assert s.lib.st_set_stream(s._h, None) == 0
        s.close()
        return t, out

    t, (q, y) = run(True, [0])
    assert np.isfinite(q).all()
    for streams in ([0], [0, other.cuda_stream]):
        t1, (q1, y1) = run(False, streams)
        assert t1 == t and np.array_equal(q1, q) and np.array_equal(y1, y)
