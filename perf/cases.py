"""The work that users of wavesim_b200 have it do, as cases that can be timed.

A case is a plain dict.  Its "kind" says which part of the package it uses:

* "solve":  one steady-state solve to tolerance (WaveSim / WaveSimVector, exec) in 2-D
            or 3-D, scalar or vector: the framework's main path;
* "angles": several plane waves on one medium in one batched solve (exec_batch);
* "pstd":   the time-domain comparison solver (PSTD, exec);
* "train":  one training step of the learned warm start (forward, backward, update).

Sizes are of the region of interest; the package adds the absorbing boundary and
rounds the grid up to an efficient length.  Media and sources are those of
wavesim_b200/workloads.py (Gaussian random media and sphere packings, 4 pixels per
wavelength; one sphere for the vector solves, 8 pixels), made from the seed.
"""
import math
import warnings

import numpy as np
import torch

import wavesim_b200 as ws
from wavesim_b200 import warmstart, workloads


# ----------------------------------------------------------------------------
# the cases
# ----------------------------------------------------------------------------
def listed():
    return [
        # a first try on a laptop-sized problem, and the inner call of an optimisation loop: latency counts
        dict(name="solve-2d-48x40", kind="solve", medium="random", ny=48, nx=40, nz=1, bw=8),
        # Green's function of a homogeneous medium (512^2 grid)
        dict(name="solve-2d-448", kind="solve", medium="uniform", ny=448, nx=448, nz=1, bw=32),
        # the disordered 2-D medium of the configurations (1024^2 grid)
        dict(name="solve-2d-960", kind="solve", medium="random", ny=960, nx=960, nz=1, bw=32),
        # a region of interest nobody rounded to a convenient size (1100 x 768 grid)
        dict(name="solve-2d-1024x700", kind="solve", medium="random", ny=1024, nx=700, nz=1, bw=32),
        # a small 3-D sphere medium (96^3 grid), as in training sets and parameter studies
        dict(name="solve-3d-64", kind="solve", medium="spheres", ny=64, nx=64, nz=64, bw=16),
        # a 3-D volume as it comes from a data set, no two sides alike (125 x 150 x 100 grid)
        dict(name="solve-3d-101x120x77", kind="solve", medium="spheres", ny=101, nx=120, nz=77, bw=11),
        # the headline 3-D sphere medium (256^3 grid)
        dict(name="solve-3d-224", kind="solve", medium="spheres", ny=224, nx=224, nz=224, bw=16),
        # Maxwell: scattering by a sphere (192^3 x 3 grid)
        dict(name="vector-160", kind="solve", medium="sphere", ny=160, nx=160, nz=160, bw=16),
        # a small Maxwell problem of uneven sides (64 x 77 x 70 x 3 grid)
        dict(name="vector-47x60x52", kind="solve", medium="sphere", ny=47, nx=60, nz=52, bw=8),
        # an angular sweep over a disordered 2-D medium in one batch (16 x 1024^2)
        dict(name="angles-16x960", kind="angles", medium="random", ny=960, nx=960, nz=1, bw=32, count=16),
        # the time-domain solver on the same kind of medium (256^2 grid)
        dict(name="pstd-2d-224", kind="pstd", medium="random", ny=224, nx=224, nz=1, bw=16),
        # a training step of the warm-start network on a crop
        dict(name="train-64", kind="train", medium="spheres", ny=64, nx=64, nz=64, bw=8),
    ]


def draw(rng):
    def side(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["2d", "2d", "2d", "3d", "3d", "3d", "vector", "vector", "angles", "pstd", "train"])
    if kind == "2d":
        medium = rng.choice(["random", "random", "random", "uniform"])
        return dict(kind="solve", medium=medium, ny=side(40, 1024), nx=side(40, 1024), nz=1, bw=rng.choice([8, 16, 25, 32]))
    if kind == "3d":
        return dict(kind="solve", medium="spheres", ny=side(40, 190), nx=side(40, 190), nz=side(40, 190),
                    bw=rng.choice([8, 11, 16]))
    if kind == "vector":
        return dict(kind="solve", medium="sphere", ny=side(40, 130), nx=side(40, 130), nz=side(40, 130),
                    bw=rng.choice([8, 11, 16]))
    if kind == "angles":
        return dict(kind="angles", medium="random", ny=side(100, 960), nx=side(100, 960), nz=1, bw=rng.choice([16, 25, 32]),
                    count=rng.randint(4, 16))
    if kind == "pstd":
        return dict(kind="pstd", medium="random", ny=side(60, 300), nx=side(60, 300), nz=1, bw=rng.choice([8, 16]))
    return dict(kind="train", medium="spheres", ny=16 * rng.randint(2, 6), nx=16 * rng.randint(2, 6), nz=16 * rng.randint(2, 6),
                bw=8)


# ----------------------------------------------------------------------------
# inputs
# ----------------------------------------------------------------------------
def medium_of(case, rng):
    """The refractive index on the region of interest."""
    shape = (case["ny"], case["nx"], case["nz"])
    if case["medium"] == "uniform":
        return np.ones(shape[:2])
    if case["medium"] == "random":  # clipped Gaussian random medium with absorption
        g = workloads.gaussian_random_field(shape[:2], workloads.PPW, rng)
        return np.clip(1.0 + 0.3 * g, 0.8, 1.6) + 0.01j
    if case["medium"] == "spheres":  # non-overlapping spheres, cut out of a cube of them
        n = workloads.sphere_medium(max(shape), rng)
        return np.ascontiguousarray(n[:shape[0], :shape[1], :shape[2]])
    # one sphere somewhere about the middle
    r = min(shape) * rng.uniform(0.1, 0.25)
    ax = [np.arange(s) + 0.5 - s * rng.uniform(0.4, 0.6) for s in shape]
    inside = ax[0][:, None, None] ** 2 + ax[1][None, :, None] ** 2 + ax[2][None, None, :] ** 2 < r ** 2
    return np.where(inside, 1.5, 1.33)


def options_of(case):
    dims = 2 if case["nz"] == 1 else 3
    o = {"boundary_widths": [case["bw"]] * dims, "energy_threshold": 1e-3}
    if case["medium"] == "sphere":
        return dict(o, **{"lambda": 0.5, "pixel_size": 0.5 / 8})
    return dict(o, **{"lambda": 1.0, "pixel_size": 1.0 / workloads.PPW})


def source_of(case, rng):
    """(values, position) of the source: a point, a beam on the left edge or a plane wave on the first face."""
    ny, nx = case["ny"], case["nx"]
    if case["medium"] == "uniform":
        return complex(rng.uniform(0.5, 1.5), rng.uniform(-0.5, 0.5)), [ny // 2 + int(rng.integers(-8, 9)), nx // 2 + int(rng.integers(-8, 9))]
    if case["medium"] == "random":
        y0 = ny * rng.uniform(0.4, 0.6)
        return np.exp(-((np.arange(ny) - y0) ** 2) / (4 * workloads.PPW) ** 2).astype(complex)[:, None], [1, 1]
    return np.full((ny, nx), 1.0, complex), [1, 1, 1]


def angles_of(case):
    """Phase advances per pixel along y of plane waves at -30 to 30 degrees."""
    return [float(v) for v in 2 * np.pi / workloads.PPW * np.sin(np.deg2rad(np.linspace(-30, 30, case["count"])))]


def training_sample(case, rng):
    """A medium and a field of the kind the network learns (a carrier with a smooth complex envelope)."""
    n = medium_of(case, rng)
    c = rng.standard_normal((2, 4, 4, 4))
    t = np.fft.ifftn(c[0] + 1j * c[1], s=n.shape) * n.size / 8
    return n, t


def prepare(case, seed):
    rng = np.random.default_rng([seed, 17])
    kind = case["kind"]
    if kind == "train":
        n, envelope = training_sample(case, rng)
        model = warmstart.WarmStart(seed=3)
        dev = model.net.dev
        x = warmstart.space_to_depth(warmstart.features(n, model.k0, model.n_bg, torch, dev), n.shape, torch)
        target = torch.from_numpy(warmstart.field_to_target(envelope, 1.0, half=True)).to(dev)
        return dict(kind=kind, model=model, x=x, target=target, vol=warmstart.roi_volume(n.shape, half=True))
    n = medium_of(case, rng)
    if kind == "pstd":
        with warnings.catch_warnings():  # its constructor says that it is there for comparison only
            warnings.simplefilter("ignore")
            sim = ws.PSTD(n, dict(options_of(case), boundary_type="ARL"))
        return dict(kind=kind, sim=sim, source=ws.Source(*source_of(case, rng)))
    sim = (ws.WaveSimVector if case["medium"] == "sphere" else ws.WaveSim)(n, options_of(case))
    sim.solver()  # uploads the medium
    if kind == "angles":
        waves = [ws.PlaneWave((case["ny"], 1), (1, 1), 1.0, (p, 0.0, 0.0)) for p in angles_of(case)]
        return dict(kind=kind, sim=sim, waves=waves)
    return dict(kind=kind, sim=sim, source=ws.Source(*source_of(case, rng)))


# ----------------------------------------------------------------------------
# the passes
# ----------------------------------------------------------------------------
def answer(E, state):
    """Field, iterations and the history of the energy (sums over a complex64 field), in an array of one size, as a program that
    collects many solves keeps it."""
    history = np.zeros(4096, np.float32)
    history[:len(state.diff_energy)] = state.diff_energy
    return {"field": E, "iterations": int(state.it), "energies": history}


def run(state):
    if state["kind"] == "train":
        net = state["model"].net
        loss = net.train_step(state["x"], state["target"], state["vol"], 2e-3)
        return {"loss": torch.tensor(loss, dtype=torch.float32),
                "gradients": [[l.gw, l.gb] for l in net.layers], "weights": [[l.w, l.b] for l in net.layers]}
    if state["kind"] == "angles":
        fields, states = state["sim"].exec_batch(state["waves"])
        return [answer(E, s) for E, s in zip(fields, states)]
    return answer(*state["sim"].exec(state["source"]))


# ----------------------------------------------------------------------------
# what a pass cannot do without
# ----------------------------------------------------------------------------
def grid_of(case):
    """Sides of the grid: the region of interest and two boundaries, rounded up to an efficient length."""
    dims = 2 if case["nz"] == 1 else 3
    return [efficient(case[k] + 2 * case["bw"]) if d < dims else 1 for d, k in enumerate(("ny", "nx", "nz"))]


def iterations_of(case):
    """About how many iterations a solve takes: a cycle has 4 (2-D) or 8 (3-D) of them, and their number grows with the grid."""
    if case["kind"] == "pstd":
        return 1500
    side = max(grid_of(case))
    if case["nz"] == 1:
        return 52 if case["medium"] == "uniform" else 230
    return 64 if case["medium"] == "sphere" else 20 + side // 2


def work(case):
    if case["kind"] == "train":
        vox = case["ny"] * case["nx"] * case["nz"] // 8
        w = (32, 64, 96, 128)
        # multiply-adds of one voxel of the first level, each coarser level having an eighth of the voxels
        conv = (64 * w[0] + w[0] * w[0] + (w[1] + w[0]) * w[0] + w[0] * w[0] + w[0] * 16
                + (w[0] * w[1] + w[1] * w[1] + (w[2] + w[1]) * w[1] + w[1] * w[1]) / 8
                + (w[1] * w[2] + w[2] * w[2] + (w[3] + w[2]) * w[2] + w[2] * w[2]) / 64
                + (w[2] * w[3] + w[3] * w[3]) / 512) * 27
        return {"bytes": vox * (64 * 2 + 16 * 4) + 3 * 4 * 2.8e6, "flops": 3 * 2.0 * vox * conv}
    N = grid_of(case)
    pts = N[0] * N[1] * N[2]
    comp = 3 if case["medium"] == "sphere" else 1
    rhs = case.get("count", 1)
    roi = case["ny"] * case["nx"] * case["nz"]
    it = iterations_of(case)
    # two 3-D transforms of 5 N log2 N and about 40 operations of the mix per iteration
    flops = it * rhs * comp * pts * (2 * 5 * math.log2(pts) + 40)
    # every iteration needs the whole increment before it: a field read and a field written each time, and the
    # medium; a grid that stays in the cache between iterations pays for them once
    state = 8.0 * pts * (3 * comp * rhs + 1)
    each = 8.0 * pts * (2 * comp * rhs + 1) if state > 100e6 else 0.0
    return {"bytes": it * each + 8.0 * pts + 8.0 * roi * comp * rhs, "flops": flops}


# ----------------------------------------------------------------------------
# the same in 64 bits, in plain torch and numpy
# ----------------------------------------------------------------------------
def efficient(n):
    """The next length whose largest prime factor is at most 11 and, of three factors or more, the second largest at most 5."""
    while True:
        f, m, p = [], n, 2
        while m > 1:
            while m % p == 0:
                f.append(p)
                m //= p
            p += 1
        if not f or (f[-1] <= 11 and (len(f) <= 2 or f[-2] <= 5)):
            return n
        n += 1


class Setup:
    """Grid, permittivity, absorbing window and wave vectors of a case, in 64 bits."""

    def __init__(self, case, n, opt):
        self.dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
        n = np.asarray(n).reshape(case["ny"], case["nx"], case["nz"])
        self.N = grid_of(case)
        self.dims = 2 if case["nz"] == 1 else 3
        self.dx, self.lam = opt["pixel_size"], opt["lambda"]
        extra = [a - b for a, b in zip(self.N, n.shape)]
        self.lo = [(e + 1) // 2 for e in extra]
        self.hi = [e // 2 for e in extra]
        self.er = self.t(np.pad(n.astype(complex) ** 2, list(zip(self.lo, self.hi)), mode="edge"))
        self.er_min, self.er_max = float(np.real(n ** 2).min()), float(np.real(n ** 2).max())
        self.roi = tuple(slice(a, N - b) for a, N, b in zip(self.lo, self.N, self.hi))
        self.window = self.t(np.ones(1))
        L = case["bw"]
        for d in range(self.dims):
            bl, br = self.lo[d], self.hi[d]
            if self.dims == 3:
                ramp = lambda B: (np.arange(1, B + 1) - 0.21) / (B + 0.66)  # noqa: E731
            else:
                t = 2 * np.pi * np.arange(2 * L - 1) / (2 * L - 2)
                nut = 0.3635819 - 0.4891775 * np.cos(t) + 0.1365995 * np.cos(2 * t) - 0.0106411 * np.cos(3 * t)
                ramp = lambda B, nut=nut: nut[:B]  # noqa: E731
            step = np.concatenate([[0.0], ramp(L - 1)]) if bl == br else ramp(L)
            w = np.concatenate([np.zeros(bl - L), step, np.ones(self.N[d] - bl - br), step[::-1], np.zeros(br - L)])
            self.window = self.window * self.axis(w, d)
        self.dp = [2 * np.pi / (self.dx * N) for N in self.N]
        # the reference's order of the wave vectors: fftshift, also for odd lengths
        self.p = [self.dp[d] * np.roll(np.arange(N) - N // 2, N // 2) for d, N in enumerate(self.N)]

    def t(self, a):
        return torch.from_numpy(np.ascontiguousarray(a)).to(self.dev)

    def axis(self, a, d):
        sh = [1, 1, 1]
        sh[d] = -1
        return self.t(a).reshape(sh)

    def source(self, values, position, comps=1):
        v = np.asarray(values, complex)
        v = v.reshape(v.shape + (1,) * (3 - v.ndim))
        S = torch.zeros([comps] + self.N, dtype=torch.complex128, device=self.dev)
        pos = [self.lo[d] + (position[d] - 1 if d < len(position) else 0) for d in range(3)]
        S[(0,) + tuple(slice(a, a + s) for a, s in zip(pos, v.shape))] = self.t(v)
        return S


def wiggles(dims):
    """The signs of the directions (y, x, z) in the iterations of a cycle, in the reference's order."""
    order = [0, 1, 3, 2] if dims == 2 else [0, 1, 2, 4, 3, 5, 6, 7]
    return [[1 - 2 * (c >> d & 1) if d < dims else 0 for d in range(3)] for c in order]


def history_of(energies):
    return torch.nn.functional.pad(torch.stack(energies), (0, 4096 - len(energies)))


def born_series(s, S, threshold, each):
    """The modified Born series for sources S [..., y, x, z]; with each, the leading axis holds solves of their own, else the
    components of one vector field.  A list of answers as run() gives them, each field on the region of interest."""
    k0 = 2 * math.pi / s.lam
    k0c = math.sqrt(0.5 * (s.er_min + s.er_max)) * k0
    V = s.er * k0 ** 2 - k0c ** 2
    eps = max(float(V.abs().max()) / 0.95, 3.0)
    gamma = 1j / eps * (V - 1j * eps) * s.window
    k02e = k0c ** 2 / eps + 1j
    cycle = wiggles(s.dims)
    nw = len(cycle)
    keep, mix = 1 - 0.7 * gamma, -0.7j * gamma ** 2
    del V
    E, dE = torch.zeros_like(S), torch.zeros_like(S)
    here = (slice(None),) + s.roi
    calc, last, diffs, found = True, None, [], [None] * (len(S) if each else 1)
    while any(f is None for f in found):
        it = len(diffs) + 1
        w = cycle[(it - 1) % nw]
        ramp = [s.axis(np.exp(0.5j * math.pi * w[d] * np.arange(N) / N), d) for d, N in enumerate(s.N)]
        ramp = ramp[0] * ramp[1] * ramp[2]
        p = [s.axis((s.p[d] - s.dp[d] * w[d] / 4) / math.sqrt(eps), d) for d in range(3)]
        P = dE + (1j / (eps * nw)) * S if it <= nw else dE
        P = torch.fft.fftn(P * ramp, dim=(1, 2, 3))
        if not each and len(S) == 3:  # components along x, y, z
            q = [p[1], p[0], p[2]]
            div = (q[0] * P[0] + q[1] * P[1] + q[2] * P[2]) / k02e
            for c in range(3):
                P[c] -= q[c] * div
            del div
        P /= p[0] ** 2 + p[1] ** 2 + (p[2] ** 2 - k02e)
        P = torch.fft.ifftn(P, dim=(1, 2, 3)) * ramp.conj()
        dE = keep * dE + mix * P
        del P
        E += dE
        if calc:
            a = dE[here].abs().square()
            last = a.sum(dim=(1, 2, 3)) if each else a.sum().reshape(1)
        diffs.append(last)
        calc = (it - 1) % 8 == 0
        if it % nw == 0:
            for r, ratio in enumerate((diffs[-1] / diffs[0]).tolist()):
                if ratio < threshold and found[r] is None:
                    F = (E[r:r + 1] if each else E)[here] / gamma[s.roi]
                    found[r] = {"field": F[0] if len(F) == 1 else F.permute(1, 2, 3, 0), "iterations": it + 1,
                                "energies": history_of([d[r] for d in diffs])}
    return found


def time_domain(s, S, threshold):
    """The pseudo-spectral time-domain stepping with the slowly switched-on source."""
    dt = 0.95 * 2 / math.sqrt(s.dims) / math.pi * s.dx * math.sqrt(s.er_min)
    per_cycle = s.lam / dt
    damp = dt * 2 * math.pi / s.lam * s.er.imag / s.er.real
    c1, c2, c3 = (damp - 2) / (damp + 2), 4 / (damp + 2), 2 * dt ** 2 / s.er.real / (damp + 2)
    lap = -(s.axis(s.p[0] ** 2, 0) + s.axis(s.p[1] ** 2, 1) + s.axis(s.p[2] ** 2, 2))

    def amplitude(cycles):
        return np.exp(-2j * math.pi * cycles) * (0.5 - 0.5 * math.cos(math.pi * min(cycles / 100, 1)))

    S = S[0]
    E, before = torch.zeros_like(S), torch.zeros_like(S)
    A, calc, diffs = 1.0, True, []
    while True:
        it = len(diffs) + 1
        A_before, A = A, complex(amplitude(it / per_cycle))
        new = c2 * E + c1 * before + c3 * (torch.fft.ifftn(lap * torch.fft.fftn(E)) + A * S)
        if calc:
            turn = complex(np.exp(1j * (np.angle(A) - np.angle(A_before))))
            last = (new - E * turn)[s.roi].abs().square().sum() / abs(A) ** 2
        diffs.append(last)
        before, E = E, new
        calc = (it - 1) % 8 == 0
        if A.real > 0.9 and float(diffs[-1] / diffs[0]) < threshold:
            F = E[s.roi] * complex(np.exp(-1j * np.angle(amplitude((it + 1) / per_cycle))))
            return {"field": F, "iterations": it + 1, "energies": history_of(diffs)}


def training_step(st):
    """Loss and gradients of the network on the inputs of a state, by autograd in 64 bits.  The weights after the step have no
    value here: its first update divides each gradient by itself, which says nothing where that is near zero."""
    net, vol = st["model"].net, st["vol"]
    wb = []
    for l in net.layers:
        w = l.w[:, :l.k].to(torch.bfloat16).double().reshape(l.cout, 3, 3, 3, l.cin).permute(0, 4, 1, 2, 3)
        wb.append((w.contiguous().requires_grad_(), l.b.double().requires_grad_()))
    F = torch.nn.functional
    layer = iter(wb)

    def conv(x, relu=True):
        w, b = next(layer)
        # one tap after the other: the library has no fast 64-bit convolution in three dimensions
        x = F.pad(x, (1, 1, 1, 1, 1, 1))
        D, H, W = (v - 2 for v in x.shape[2:])
        y = 0
        for t in range(27):
            z, r, c = t // 9, t // 3 % 3, t % 3
            y = y + torch.einsum("oi,bizyx->bozyx", w[:, :, z, r, c], x[:, :, z:z + D, r:r + H, c:c + W])
        y = y + b[:, None, None, None]
        return torch.relu(y) if relu else y

    def up(a, skip):
        return torch.cat([F.interpolate(a, scale_factor=2, mode="nearest"), skip], dim=1)

    x = st["x"].double().reshape(*vol, -1).permute(0, 4, 1, 2, 3)
    e1 = conv(conv(x))
    e2 = conv(conv(F.avg_pool3d(e1, 2)))
    e3 = conv(conv(F.avg_pool3d(e2, 2)))
    b4 = conv(conv(F.avg_pool3d(e3, 2)))
    d3 = conv(conv(up(b4, e3)))
    d2 = conv(conv(up(d3, e2)))
    d1 = conv(conv(up(d2, e1)))
    out = conv(d1, relu=False).permute(0, 2, 3, 4, 1).reshape(st["target"].shape)
    loss = (out - st["target"].double()).square().mean()
    loss.backward()
    grads = []
    for l, (w, b) in zip(net.layers, wb):
        g = torch.zeros(l.cout, l.kp, dtype=torch.float64, device=w.device)
        g[:, :l.k] = w.grad.permute(0, 2, 3, 4, 1).reshape(l.cout, l.k)
        grads.append([g, b.grad])
    return {"loss": loss.detach(), "gradients": grads, "weights": [[None, None] for _ in grads]}


def exact(case, seed):
    if case["kind"] == "train":
        return training_step(prepare(case, seed))
    rng = np.random.default_rng([seed, 17])
    s = Setup(case, medium_of(case, rng), options_of(case))
    if case["kind"] == "angles":
        y = np.arange(case["ny"])
        S = torch.cat([s.source(np.exp(1j * p * y)[:, None], [1, 1]) for p in angles_of(case)])
        return born_series(s, S, 1e-3, True)
    S = s.source(*source_of(case, rng), comps=3 if case["medium"] == "sphere" else 1)
    if case["kind"] == "pstd":
        return time_domain(s, S, 1e-3)
    return born_series(s, S, 1e-3, False)[0]
