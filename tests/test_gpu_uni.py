"""The run-time scheduled kernels (wavesim_b200/csrc/ws_uni.cuh) against the
generic kernels and the FP32 oracle where they can go wrong: lines of two,
three and four stages, odd and even last radices (padding), every radix class,
rows that do not fill a tile, columns that do not fill a block, one wiggle (a
periodic grid) and eight, three components, and next to a fast inner pass.

A dozen iterations of single-precision transforms of these lengths differ by a
few 1e-7; 1e-5 leaves room for that and none for a wrong element."""

import numpy as np
import pytest

from oracle import mbs_oracle as ref

pytestmark = pytest.mark.gpu

TOL = 1e-5

CASES = {
    # name: (roi shape, boundary widths (0: periodic, the size is taken as it is), vector)
    "2d_4x6_one_wiggle": ((4, 6), [0, 0], False),
    "2d_45x60": ((33, 42), [6, 8], False),
    "2d_26x39": ((26, 39), [0, 0], False),
    "2d_1100x21": ((1068, 21), [16, 0], False),
    "2d_four_stages_2401x18": ((2401, 18), [0, 0], False),
    "2d_18x2401": ((18, 2401), [0, 0], False),
    "2d_64_columns_x_56": ((48, 40), [8, 8], False),
    "2d_225x256": ((225, 256), [0, 0], False),
    "3d_27x25x50": ((15, 13, 38), [6, 6, 6], False),
    "3d_125x24x33": ((109, 12, 21), [8, 6, 6], False),
    "3d_15x198x243": ((15, 198, 243), [0, 0, 0], False),
    "3d_64_planes_z_50": ((48, 48, 38), [8, 8, 6], False),
    "3d_vector_26x30x21": ((26, 18, 9), [0, 6, 6], True),
    "3d_vector_63x16x105": ((47, 16, 89), [8, 0, 8], True),
    "2d_vector_45x60": ((33, 42), [6, 8], True),
    "2d_vector_64x50": ((64, 50), [0, 0], True),
}


def rel(a, b):
    return float(np.linalg.norm(np.ravel(a) - np.ravel(b)) / np.linalg.norm(np.ravel(b)))


@pytest.mark.parametrize("name", list(CASES))
def test_uni_matches_generic_and_oracle(gpu, name, monkeypatch):
    import wavesim_b200 as ws
    shape, bw, vector = CASES[name]
    rng = np.random.default_rng(11)
    n = 1.2 + 0.2 * rng.random(shape) + 0.005j
    iters = 8 if len(shape) == 3 else 12
    opt = {"lambda": 1.0, "pixel_size": 0.125 if vector else 0.25, "boundary_widths": bw, "energy_threshold": 1e-99,
           "max_iterations": iters}
    val = rng.standard_normal(shape[:2]) + 1j * rng.standard_normal(shape[:2])
    pos = [1] * len(shape) + [1] * (3 - len(shape)) + ([2] if vector else [])

    def product():
        sim = (ws.WaveSimVector if vector else ws.WaveSim)(n, opt)
        E, st = sim.exec(ws.Source(val, pos))
        sim.close()
        return E, st

    E, st = product()
    monkeypatch.setenv("WAVESIM_B200_PATH", "generic")
    Eg, sg = product()
    Eo, so = (ref.WaveSimVector if vector else ref.WaveSim)(n, opt).exec(ref.Source(val, pos), max_iterations=iters)
    assert st.it == sg.it == so.it
    assert rel(E, Eg) < TOL and rel(E, Eo) < TOL, (rel(E, Eg), rel(E, Eo))
    np.testing.assert_allclose(st.diff_energy, so.diff_energy, rtol=2e-4)


LOOPS = {
    # the loop in one launch: on a cluster of 16 blocks, at the edges of its tiles, with E' in shared
    # memory and not, and on a grid that has compile-time kernels for its launched passes
    "64x56_cluster": ((48, 40), [8, 8]),
    "4x6": ((4, 6), [0, 0]),
    "160x264": ((96, 200), [32, 32]),
    "225x150": ((225, 150), [0, 0]),
    "1100x768_E_in_global": ((1068, 736), [16, 16]),
    "512x512_fast_passes": ((448, 448), [32, 32]),
}


def loop_sim(ws, name, **more):
    shape, bw = LOOPS[name]
    rng = np.random.default_rng(5)
    n = 1.1 + 0.2 * rng.random(shape) + 0.01j
    opt = {"lambda": 1.0, "pixel_size": 0.25, "boundary_widths": bw, "energy_threshold": 1e-3, "max_iterations": 40}
    opt.update(more)
    return ws.WaveSim(n, opt), ws.Source(np.ones((shape[0], 1)) + 0.4j, [1, 1])


@pytest.mark.parametrize("name", list(LOOPS))
@pytest.mark.parametrize("use_graph", [True, False])
def test_loop_in_one_launch_is_bit_identical(gpu, name, use_graph, monkeypatch):
    """One launch for the whole loop (use_graph) or per cycle, against one launch per pass."""
    import wavesim_b200 as ws
    got = []
    for fuse in ("1", "0"):
        monkeypatch.setenv("WAVESIM_B200_FUSE", fuse)
        sim, src = loop_sim(ws, name, use_graph=use_graph)
        got.append(sim.exec(src))
        sim.close()
    (E, st), (Eu, su) = got
    assert st.it == su.it
    np.testing.assert_array_equal(st.diff_energy, su.diff_energy)
    np.testing.assert_array_equal(E, Eu)


def test_loop_over_several_launches_and_batches(gpu):
    """More cycles than one launch takes; and several right-hand sides in one launch."""
    import wavesim_b200 as ws
    sim, src = loop_sim(ws, "64x56_cluster", energy_threshold=1e-99, max_iterations=2200)
    E, st = sim.exec(src)
    sim.use_graph = False  # a launch per cycle
    Eh, sh = sim.exec(src)
    assert st.it == sh.it == 2201
    np.testing.assert_array_equal(st.diff_energy, sh.diff_energy)
    np.testing.assert_array_equal(E, Eh)
    sim.close()
    sim, src = loop_sim(ws, "64x56_cluster", energy_threshold=1e-6, max_iterations=4000)
    sources = [src, ws.Source(1.0, [24, 20]), src]
    Eb, sb = sim.exec_batch(sources)
    for s, e, t in zip(sources, Eb, sb):
        E1, s1 = sim.exec(s)
        assert t.it == s1.it and t.converged
        np.testing.assert_array_equal(e, E1)
    sim.close()


@pytest.mark.filterwarnings("ignore:The PSTD code")
@pytest.mark.parametrize("shape,bw", [((4, 6), [0, 0]), ((48, 40), [8, 8]), ((33, 150), [6, 0]), ((240, 240), [8, 8]),
                                      ((736, 1068), [16, 16])])
def test_pstd_in_one_launch_matches_launched_passes(gpu, shape, bw, monkeypatch):
    """300 steps (two launches of at most 256), against the generic kernels' five launches a step.  Each step rounds to a
    few 1e-7; their random sum over 300 steps is 5e-6, and 5e-5 leaves ten times that."""
    import wavesim_b200 as ws
    n = 1.0 + 0.2 * np.random.default_rng(2).random(shape) + 0.02j
    opt = {"lambda": 1.0, "pixel_size": 0.25, "boundary_widths": bw, "boundary_type": "ARL", "energy_threshold": 1e-30,
           "source_amplitude": lambda c: np.exp(-2.0j * np.pi * c)}
    got = []
    for path in ("", "generic"):
        monkeypatch.setenv("WAVESIM_B200_PATH", path)
        p = ws.PSTD(n, opt)
        got.append(p.exec(ws.Source(np.ones((shape[0], 1)) + 0.5j, [1, 2]), max_iterations=300))
        p.close()
    (E, st), (Eg, sg) = got
    assert st.it == sg.it
    assert rel(E, Eg) < 5e-5, rel(E, Eg)
    np.testing.assert_allclose(st.diff_energy, sg.diff_energy, rtol=1e-3)


@pytest.mark.parametrize("shape,bw,count", [((480, 960), [16, 32], 5), ((256, 448), [32, 32], 16)])
def test_batched_x_pencils_match_single_solves(gpu, shape, bw, count):
    """Batches of 2-D grids of 1024 and 512 points along x run their x pencils through the tensor-copy pipeline
    (tma::kt_pencil with D3 = false), single solves do not."""
    import wavesim_b200 as ws
    n = 1.1 + 0.2 * np.random.default_rng(8).random(shape) + 0.01j
    sim = ws.WaveSim(n, {"lambda": 1.0, "pixel_size": 0.25, "boundary_widths": bw, "energy_threshold": 1e-99,
                         "max_iterations": 12})
    waves = [ws.PlaneWave((shape[0], 1), (1, 1), 1.0, (0.05 * k, 0.0, 0.0)) for k in range(count)]
    E, st = sim.exec_batch(waves)
    for k in (0, count - 1):
        E1, s1 = sim.exec(ws.Source(waves[k].values()[..., 0], [1, 1]))
        assert st[k].it == s1.it
        assert rel(E[k], E1) < TOL, rel(E[k], E1)
        np.testing.assert_allclose(st[k].diff_energy, s1.diff_energy, rtol=2e-4)
    sim.close()
