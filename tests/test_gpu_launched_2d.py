"""The launched passes of 2-D grids, where single solves run the loop in one launch instead."""
import ctypes as C

import numpy as np
import pytest

from oracle import mbs_oracle as ref

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


def test_a_tuned_layout_leaves_the_loop_in_one_launch(gpu):
    import wavesim_b200 as ws
    from wavesim_b200 import _lib
    from wavesim_b200.autotune import set_layout
    n = 1.1 + 0.2 * np.random.default_rng(3).random((96, 80)) + 0.01j
    sim = ws.WaveSim(n, {"lambda": 1.0, "pixel_size": 0.25, "boundary_widths": [16, 16], "energy_threshold": 1e-3})
    src = ws.Source(1.0, [48, 40])
    E0, s0 = sim.exec(src)
    h = sim.solver()
    for choose in (lambda: set_layout(sim, [2, 2, 0, 0, 0, 0, 0]), lambda: set_layout(sim, [0, 2, 0, 0, 4, 0, 0]),
                   lambda: _lib.check(_lib.lib.ws_solver_autotune(h, 4, None, None, None))):
        choose()
        assert _lib.lib.ws_solver_loop_in_one_launch(h) == 1
        E1, s1 = sim.exec(src)
        assert s1.it == s0.it
        np.testing.assert_array_equal(E1, E0)
    sim.close()


@pytest.mark.parametrize("shape,bw,room", [((96, 200), [32, 32], 131), ((96, 200), [32, 32], 0), ((48, 40), [8, 8], 15),
                                           ((48, 40), [8, 8], 7)])
def test_without_room_for_the_loop_the_passes_are_launched(gpu, shape, bw, room, monkeypatch):
    """160 x 264 has 132 column tiles, 64 x 56 has 14 (and 16 tiles of pencils): with fewer blocks at a time than column
    tiles the solve runs the launched passes; with fewer than all tiles the loop is no cluster.  A dozen iterations of
    single precision differ by a few 1e-7."""
    import wavesim_b200 as ws
    from wavesim_b200 import _lib
    n = 1.1 + 0.2 * np.random.default_rng(5).random(shape) + 0.01j
    opt = {"lambda": 1.0, "pixel_size": 0.25, "boundary_widths": bw, "energy_threshold": 1e-99, "max_iterations": 12}
    src = ws.Source(np.ones((shape[0], 1)) + 0.4j, [1, 1])
    sim = ws.WaveSim(n, opt)
    assert _lib.lib.ws_solver_loop_in_one_launch(sim.solver()) == 1
    E0, s0 = sim.exec(src)
    sim.close()
    monkeypatch.setenv("WAVESIM_B200_LOOP", str(room))
    sim = ws.WaveSim(n, opt)
    assert _lib.lib.ws_solver_loop_in_one_launch(sim.solver()) == (1 if room == 15 else 0)
    E1, s1 = sim.exec(src)
    sim.close()
    assert s1.it == s0.it
    assert np.linalg.norm(E1 - E0) < 1e-5 * np.linalg.norm(E0)
    monkeypatch.delenv("WAVESIM_B200_LOOP")


@pytest.mark.filterwarnings("ignore:The PSTD code")
def test_pstd_without_room_for_its_loop(gpu, monkeypatch):
    import wavesim_b200 as ws
    n = 1.0 + 0.2 * np.random.default_rng(2).random((60, 70)) + 0.02j
    opt = {"lambda": 1.0, "pixel_size": 0.25, "boundary_widths": [8, 8], "boundary_type": "ARL", "energy_threshold": 1e-30}
    got = []
    for room in ("", "9"):
        if room:
            monkeypatch.setenv("WAVESIM_B200_LOOP", room)
        p = ws.PSTD(n, opt)
        got.append(p.exec(ws.Source(np.ones((60, 1)), [1, 2]), max_iterations=100)[0])
        p.close()
    assert np.linalg.norm(got[1] - got[0]) < 5e-5 * np.linalg.norm(got[0])


# The compile-time kernels of 2-D grids: single solves of these sizes run the loop in one launch, batches too large for
# it still run these passes.
FAST = {"64": ((32, 32), [16, 16]), "128x256": ((96, 224), [16, 16]), "512": ((448, 448), [32, 32]),
        "320": ((256, 256), [32, 32]), "448": ((384, 384), [32, 32]), "576": ((512, 512), [32, 32]),
        "192": ((160, 160), [16, 16]), "320x100": ((256, 68), [32, 16]), "256x192": ((224, 160), [16, 16]),
        "512x120": ((448, 100), [32, 10])}


@pytest.mark.parametrize("name", list(FAST))
def test_compile_time_kernels_without_the_loop(gpu, name, monkeypatch):
    """Against the FP32 oracle, and the fused column pass against K1 and K3 as kernels of their own, bit for bit.  16
    iterations of single precision differ by a few 1e-7; 1e-5 leaves none for a wrong element."""
    import wavesim_b200 as ws
    from wavesim_b200 import _lib
    shape, bw = FAST[name]
    rng = np.random.default_rng(7)
    n = 1.2 + 0.2 * rng.random(shape) + 0.005j
    opt = {"lambda": 1.0, "pixel_size": 0.25, "boundary_widths": bw, "energy_threshold": 1e-99, "max_iterations": 16}
    val = rng.standard_normal(shape) + 1j * rng.standard_normal(shape)
    monkeypatch.setenv("WAVESIM_B200_LOOP", "0")
    got = []
    for fuse in ("1", "0"):
        monkeypatch.setenv("WAVESIM_B200_FUSE", fuse)
        sim = ws.WaveSim(n, opt)
        assert _lib.lib.ws_solver_loop_in_one_launch(sim.solver()) == 0
        assert _lib.lib.ws_solver_fused(sim.solver()) == int(fuse)
        got.append(sim.exec(ws.Source(val, [1, 1])))
        sim.close()
    (E, st), (Eu, su) = got
    Eo, so = ref.WaveSim(n, opt).exec(ref.Source(val, [1, 1, 1]), max_iterations=16)
    assert st.it == su.it == so.it
    np.testing.assert_array_equal(E, Eu)
    np.testing.assert_array_equal(st.diff_energy, su.diff_energy)
    Eo = Eo.reshape(E.shape)
    assert np.linalg.norm(E - Eo) < 1e-5 * np.linalg.norm(Eo)
    np.testing.assert_allclose(st.diff_energy, so.diff_energy, rtol=2e-4)
