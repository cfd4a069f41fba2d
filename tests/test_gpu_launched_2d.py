"""The launched passes of 2-D grids, where single solves run the loop in one launch instead."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_queries_are_about_the_launched_passes(gpu):
    """48 x 64: compile-time x pencils, but no column kernel, so the launched passes are the generic K1, pencils, K3 -
    not fused, whatever the loop in one launch does."""
    import wavesim_b200 as ws
    from wavesim_b200 import _lib
    n = 1.1 + 0.1 * np.random.default_rng(3).random((48, 64)) + 0.01j
    sim = ws.WaveSim(n, {"lambda": 1.0, "pixel_size": 0.25, "boundary_widths": [0, 0], "energy_threshold": 1e-3})
    src = ws.Source(1.0, [24, 32])
    E0, s0 = sim.exec(src)
    h = sim.solver()
    ms, by, ms3, by3 = C.c_float(), C.c_double(), (C.c_float * 3)(), (C.c_double * 3)()
    for _ in range(2):
        assert _lib.lib.ws_solver_fused(h) == 0
        assert _lib.lib.ws_solver_launches_per_iteration(h) == 3
        assert _lib.lib.ws_solver_time_fused(h, 4, C.byref(ms), C.byref(by)) == _lib.WS_ERR_UNSUPPORTED
        assert _lib.lib.ws_solver_time_split(h, 4, ms3, by3) == _lib.WS_ERR_UNSUPPORTED
        assert _lib.lib.ws_solver_time_kernels(h, 4, ms3, by3) == _lib.WS_OK and all(v > 0 for v in ms3)
        E1, s1 = sim.exec(src)
        assert s1.it == s0.it
        np.testing.assert_array_equal(E1, E0)
    sim.close()
