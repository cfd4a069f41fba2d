"""Converged solves on the run-time scheduled kernels (wavesim_b200/csrc/ws_uni.cuh)
against the FP64 oracle run on the solver's own single-precision tables (gamma,
p, k02e, epsilon), so that what differs is the solver's arithmetic alone.

What a solve adds up coherently is the transforms' round-trip gain.  Taken out
to first order by position and by frequency, 1e-8 of it is left (the constants'
cross terms); each 4e-8 moves the field of a disordered 2-D solve by 1.4e-6 and
its energies by 8e-7 (in 200 iterations, in proportion), so 3.5e-7 and 2e-7.
The rest is rounding without a preferred sign: the sum E' over 100 additions
3.5e-7, ramps 3e-7, transforms and mix 6e-7 together, on the energies 2e-7.
In squares that is below 1.2e-6 and 4e-7.  (Uncorrected, the first five cases'
gains are 3e-8 to 1.4e-7.)"""

import numpy as np
import pytest

from oracle import mbs_oracle as ref

pytestmark = pytest.mark.gpu

CASES = {
    # name: (roi, boundary widths, vector): the grids are the names
    "165x400": ((133, 368), [16, 16], False),
    "81x360": ((65, 344), [8, 8], False),
    "60x270": ((44, 254), [8, 8], False),
    "375x105": ((343, 73), [16, 16], False),
    "252x432": ((220, 400), [16, 16], False),
    "54x45x50": ((38, 29, 34), [8, 8, 8], False),
    "vector_42x45x40": ((26, 29, 24), [8, 8, 8], True),
}


def medium(shape, vector):
    from wavesim_b200.workloads import gaussian_random_field
    rng = np.random.default_rng(31)
    if len(shape) == 2:
        return np.clip(1.0 + 0.3 * gaussian_random_field(shape, 4, rng), 0.8, 1.6) + 0.01j
    ax = [np.arange(s) - 0.45 * s for s in shape]
    r2 = ax[0][:, None, None] ** 2 + ax[1][None, :, None] ** 2 + ax[2][None, None, :] ** 2
    return np.where(r2 < (0.2 * min(shape)) ** 2, 1.5, 1.33)


def in_64_bits(n, opt, sim, source, vector):
    """The oracle in double precision with sim's tables, ramps of modulus 1."""
    o = (ref.WaveSimVector if vector else ref.WaveSim)(n, dict(opt, single_precision=False))
    assert tuple(o.N[:3]) == tuple(int(v) for v in sim.N[:3])
    o.gamma = sim.gamma.astype(np.complex128)
    o.k02e = complex(sim.k02e)
    o.epsilon = float(sim.epsilon)
    for a, b in zip(o.wiggles, sim.wiggles):
        a.pxe, a.pye, a.pze = (np.asarray(v, np.float64) for v in (b.pxe, b.pye, b.pze))
    return o.exec(source)


@pytest.mark.parametrize("name", list(CASES))
def test_converged_field_and_energies_against_64_bits(gpu, name):
    import wavesim_b200 as ws
    shape, bw, vector = CASES[name]
    n = medium(shape, vector)
    opt = {"lambda": 1.0, "pixel_size": 0.125 if vector else 0.25, "boundary_widths": bw, "energy_threshold": 1e-3}
    val = np.exp(-((np.arange(shape[0]) - 0.45 * shape[0]) / 16) ** 2)[:, None] if len(shape) == 2 else np.ones(shape[:2])
    pos = [1] * len(shape)
    sim = (ws.WaveSimVector if vector else ws.WaveSim)(n, opt)
    assert name.endswith("x".join(str(int(v)) for v in sim.N[:len(shape)]))
    E, st = sim.exec(ws.Source(val, pos))
    Eo, so = in_64_bits(n, opt, sim, ref.Source(val, pos + [1] * (3 - len(shape)) + ([1] if vector else [])), vector)
    sim.close()
    assert st.it == so.it and st.converged
    field = np.linalg.norm(np.ravel(E - Eo)) / np.linalg.norm(np.ravel(Eo))
    d = np.asarray(so.diff_energy)
    energies = np.linalg.norm(st.diff_energy - d) / np.linalg.norm(d)
    print(name, st.it, "%.2e %.2e" % (field, energies))
    assert field < 1.2e-6 and energies < 4e-7, (field, energies)
