"""The barrier of the loops in one launch (uni::grid_barrier) has a bound that
ws_solver_set_wait_limit (ws_pstd_set_wait_limit) reaches: with a limit of one clock the blocks give up,
set the error flag and return; the solve reports it, and the next one, with the
default limit, is the ordinary solve bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("use_graph", [True, False])
def test_loop_barrier_runs_out_and_reports(gpu, use_graph):
    import wavesim_b200 as ws
    from wavesim_b200 import WaveSimError, _lib
    shape = (96, 200)  # 160 x 264: more tiles than one cluster takes
    n = 1.1 + 0.2 * np.random.default_rng(5).random(shape) + 0.01j
    sim = ws.WaveSim(n, {"lambda": 1.0, "pixel_size": 0.25, "boundary_widths": [32, 32], "energy_threshold": 1e-3,
                         "use_graph": use_graph})
    src = ws.Source(np.ones((shape[0], 1)) + 0.4j, [1, 1])
    E0, s0 = sim.exec(src)
    for _ in range(2):
        _lib.check(_lib.lib.ws_solver_set_wait_limit(sim.solver(), 1))
        with pytest.raises(WaveSimError) as e:
            sim.exec(src)
        assert e.value.status == _lib.WS_ERR_CUDA
        assert b"timed out" in _lib.lib.ws_last_error()
        _lib.check(_lib.lib.ws_solver_set_wait_limit(sim.solver(), 0))
        E1, s1 = sim.exec(src)
        assert s1.it == s0.it
        np.testing.assert_array_equal(s1.diff_energy, s0.diff_energy)
        np.testing.assert_array_equal(E1, E0)
    sim.close()


@pytest.mark.filterwarnings("ignore:The PSTD code")
def test_pstd_runs_again_after_its_barrier_ran_out(gpu):
    import wavesim_b200 as ws
    from wavesim_b200 import WaveSimError, _lib
    shape = (120, 150)
    n = 1.0 + 0.2 * np.random.default_rng(2).random(shape) + 0.02j
    p = ws.PSTD(n, {"lambda": 1.0, "pixel_size": 0.25, "boundary_widths": [8, 8], "boundary_type": "ARL",
                    "energy_threshold": 1e-2})
    src = ws.Source(np.ones((shape[0], 1)), [1, 2])
    E0, s0 = p.exec(src)
    _lib.check(_lib.lib.ws_pstd_set_wait_limit(p._handle(), 1))
    with pytest.raises(WaveSimError) as e:
        p.exec(src)
    assert e.value.status == _lib.WS_ERR_CUDA and b"timed out" in _lib.lib.ws_last_error()
    _lib.check(_lib.lib.ws_pstd_set_wait_limit(p._handle(), 0))
    for _ in range(2):
        E1, s1 = p.exec(src)
        assert s1.it == s0.it
        np.testing.assert_array_equal(E1, E0)
    p.close()
