"""What a user of the framework runs, as timed cases: particle-mesh runs of single peaks over the
range of mesh sizes, the drop-in step surface, ensembles through the batch API and the device
initial conditions.

Every pass starts from the same inputs (particles are loaded at its start), so it can be repeated.
Engine states are returned in single precision, the precision the engine holds them in, and
positions as displacements from the lattice, so that a particle on the periodic seam is not a box
length away from itself.
"""
from __future__ import annotations

import math
import types

import numpy as np
import torch

from pbh_b200 import _lib
from pbh_b200.batch import Ensemble
from pbh_b200.engine import Engine, PeakConfig
from pbh_b200.ic import KIND_GAUSS, KIND_ZETA, make_particles
from pbh_b200.recipe import PeakSpec

H_I = 5.0
MESHES = (32, 64, 128, 256)
RATIO = 100.0 ** (1.0 / 150.0) - 1.0      # 150 steps uniform in ln a over the factor 100 of a recipe run
R_BAR = (0.10 * 0.09 * 0.08) ** (1.0 / 3.0)


def _run(name, N, Np, steps, a0=10.0, gradient="spectral", smooth=0.0, tile=0, schedule="ratio", rate=RATIO):
    return dict(name=name, kind="run", N=N, Np=Np, steps=steps, a0=a0, gradient=gradient, smooth=smooth, tile=tile,
                schedule=schedule, rate=rate)


def listed():
    return [
        # PM3D.step on the smallest recipe mesh, the density back after every step: launches and
        # host round trips.
        dict(name="steps_32", kind="steps", N=32, Np=32, steps=10, a0=10.0, gradient="spectral", smooth=0.0, tile=0,
             rate=0.02),
        # Stretches of single runs of the recipe's mesh sizes, from a tenth of the way to the end
        # (load, steps from one captured graph, read back).
        _run("run_64", 64, 64, 24),
        _run("run_128", 128, 128, 24),
        # The driver's default run: twice as many cells as particles per axis, smoothed forces,
        # da = 0.02 a.
        _run("driver_128", 128, 64, 24, smooth=2.0, schedule="frac", rate=0.02),
        # Finite-difference gradient, a lattice that does not divide the mesh, small super-tiles.
        _run("ragged_64", 64, 75, 16, gradient="fd4", smooth=1.0, tile=8),
        # The plain 256^3 run, and the same through collapse (dense super-tiles, relayouts).
        _run("run_256", 256, 256, 24),
        _run("collapse_256", 256, 256, 16, a0=60.0),
        # The large single run.
        _run("run_512", 512, 512, 12),
        # Many small peaks at once, as a request loop's slots or a parameter scan hold them.
        dict(name="scan_small", kind="ensemble", n32=24, n64=16, n128=0, n256=0, steps=112),
        # The mixed ensemble of 32^3 to 256^3 peaks: noise fields to final densities.
        dict(name="ensemble", kind="ensemble", n32=4, n64=4, n128=4, n256=3, steps=112),
        # Initial conditions alone: a recipe peak with noise, and a curvature profile with a
        # band-limited tail on a lattice finer than the mesh.
        dict(name="ic_256", kind="ic", profile="gauss", N=256, Np=256, noise=True),
        dict(name="ic_profile_64", kind="ic", profile="zeta", N=64, Np=80, noise=True),
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    pick = rng.random()
    N = rng.choice(MESHES)
    if pick < 0.6:
        Np = _logint(rng, N / 2, N * 1.2)
        c = _run("", N, Np, rng.randint(8, 24), a0=math.exp(rng.uniform(math.log(5.0), math.log(60.0))),
                 gradient=rng.choice(["spectral", "spectral", "fd2", "fd4"]), smooth=rng.choice([0.0, 0.0, 1.0, 2.0]),
                 tile=rng.choice([0, 0, 0, 4, 8]), schedule=rng.choice(["ratio", "frac"]),
                 rate=rng.uniform(0.015, 0.05))
        del c["name"]
        return c
    if pick < 0.7:
        N = rng.choice([16, 32, 64])
        return dict(kind="steps", N=N, Np=_logint(rng, N / 2, N * 1.2), steps=rng.randint(4, 12), a0=math.exp(rng.uniform(math.log(5.0), math.log(60.0))),
                    gradient="spectral", smooth=rng.choice([0.0, 2.0]), tile=0, rate=rng.uniform(0.015, 0.05))
    if pick < 0.8:
        return dict(kind="ensemble", n32=rng.randint(0, 16), n64=rng.randint(1, 16), n128=rng.randint(0, 6),
                    n256=rng.randint(0, 2), steps=rng.randint(64, 120))
    return dict(kind="ic", profile=rng.choice(["gauss", "zeta"]), N=N, Np=_logint(rng, N / 2, N * 1.2),
                noise=rng.random() < 0.7)


# ------------------------------------------------------------------------------ inputs
def _params(seed, k=0):
    """Shape, amplitude and collapse time of peak k of a seed, over the recipe's ranges."""
    g = np.random.default_rng([int(seed), int(k)])
    e, p = g.uniform(0.05, 0.3), g.uniform(-0.1, 0.1)
    lam = np.array([1.0 + 3.0 * e + p, 1.0 - 2.0 * p, 1.0 - 3.0 * e + p]) / 3.0
    ax = lam ** -0.5
    ax = ax / np.prod(ax) ** (1.0 / 3.0)
    a_c = math.exp(g.uniform(math.log(0.3), 0.0))
    return dict(e=e, p=p, axes=ax, R=tuple(float(v) for v in R_BAR * ax), delta0=1.4 / (100.0 * a_c), mu=g.uniform(0.05, 0.15))


def _normals(seed, k, N):
    g = torch.Generator(device="cuda").manual_seed(int(seed) * 1009 + int(k))
    return torch.randn((N, N, N), generator=g, device="cuda", dtype=torch.float64)


def _profile():
    """A cubic piecewise polynomial of the curvature profile exp(-r^2/2) on [0, 6], in the layout
    of scipy's CubicSpline (x and c)."""
    x = np.linspace(0.0, 6.0, 241)
    y, s = np.exp(-0.5 * x * x), -x * np.exp(-0.5 * x * x)
    h = np.diff(x)
    m = np.diff(y) / h
    c = np.stack([(s[:-1] + s[1:] - 2 * m) / h ** 2, (3 * m - 2 * s[:-1] - s[1:]) / h, s[:-1], y[:-1]])
    return types.SimpleNamespace(x=x, c=c)


# The Zel'dovich particles of a field in plain torch, in 64 bits.
def _kgrid(N, L):
    k1 = 2 * math.pi * torch.fft.fftfreq(N, d=L / N, dtype=torch.float64, device="cuda")
    kz = 2 * math.pi * torch.fft.rfftfreq(N, d=L / N, dtype=torch.float64, device="cuda")
    return k1.view(-1, 1, 1), k1.view(1, -1, 1), kz.view(1, 1, -1)


def _corners(X, N, dx):
    g = X / dx - 0.5
    lo = torch.floor(g)
    f = g - lo
    lo = lo.to(torch.int64)
    i0, i1 = torch.remainder(lo, N), torch.remainder(lo + 1, N)
    for ix, wx in ((i0[:, 0], 1 - f[:, 0]), (i1[:, 0], f[:, 0])):
        for iy, wy in ((i0[:, 1], 1 - f[:, 1]), (i1[:, 1], f[:, 1])):
            for iz, wz in ((i0[:, 2], 1 - f[:, 2]), (i1[:, 2], f[:, 2])):
                yield (ix * N + iy) * N + iz, wx * wy * wz


def _parts(n, size=1 << 24):
    return [slice(i, min(n, i + size)) for i in range(0, n, size)]


def _gather(F, X, N, dx):
    out = torch.empty(X.shape[0], dtype=torch.float64, device="cuda")
    flat = F.reshape(-1)
    for s in _parts(X.shape[0]):
        out[s] = sum(flat[i] * w for i, w in _corners(X[s], N, dx))
    return out


def _lattice(Np, L):
    q = (torch.arange(Np, dtype=torch.float64, device="cuda") + 0.5) * (L / Np)
    return torch.stack(torch.meshgrid(q, q, q, indexing="ij"), dim=-1).reshape(-1, 3)


def _field(N, L, P, profile, noise, tail):
    """Linear density spectrum of a peak (noise: standard normals or None) and its k grid."""
    x = (torch.arange(N, dtype=torch.float64, device="cuda") + 0.5) * (L / N) - L / 2
    X2, Y2, Z2 = x.view(-1, 1, 1) ** 2, x.view(1, -1, 1) ** 2, x.view(1, 1, -1) ** 2
    kx, ky, kz = _kgrid(N, L)
    k2 = kx ** 2 + ky ** 2 + kz ** 2
    k2[0, 0, 0] = 1.0
    if profile == "zeta":
        A, sp = P["axes"], _profile()
        r = torch.sqrt(X2 / A[0] ** 2 + Y2 / A[1] ** 2 + Z2 / A[2] ** 2).clamp_(max=float(sp.x[-1]))
        i = (r / 0.025).to(torch.int64).clamp_(max=len(sp.x) - 2)
        xs, c = torch.tensor(sp.x, device="cuda"), torch.tensor(sp.c, device="cuda")
        t = r - xs[i]
        i = i - (t < 0).to(torch.int64)
        t = r - xs[i]
        dk = torch.fft.rfftn(P["mu"] * (((c[0][i] * t + c[1][i]) * t + c[2][i]) * t + c[3][i]))
        if noise is not None:
            kk = torch.sqrt(k2)
            kk[0, 0, 0] = 0.0
            rms, k1, kb = tail
            band = (kk >= k1) & (kk <= kb)
            pw = torch.where(band, 2 * math.pi ** 2 * rms ** 2 / (kk.clamp(min=1e-30) ** 3 * math.log(kb / k1)), 0.0)
            dk += torch.fft.rfftn(noise) * torch.sqrt(pw * N ** 3 / L ** 3)
        dk *= 0.4 * k2 / H_I ** 2
    else:
        R = P["R"]
        dk = torch.fft.rfftn(P["delta0"] * torch.exp(-(X2 / (2 * R[0] ** 2) + Y2 / (2 * R[1] ** 2) + Z2 / (2 * R[2] ** 2))))
        if noise is not None:
            nk = torch.fft.rfftn(noise) / torch.sqrt(k2)
            nk[0, 0, 0] = 0.0
            dk += nk * (0.01 * P["delta0"] / torch.fft.irfftn(nk, s=(N, N, N)).std(correction=0))
    dk[0, 0, 0] = 0.0
    return dk, (kx, ky, kz, k2)


def _displacements(N, Np, L, dk, grid):
    kx, ky, kz, k2 = grid
    q = _lattice(Np, L)
    d = torch.empty_like(q)
    for c, kc in enumerate((kx, ky, kz)):
        d[:, c] = _gather(torch.fft.irfftn(1j * kc * dk / k2, s=(N, N, N)), q, N, L / N)
    return q, d


def _particles(case, seed):
    """Positions and momenta of a peak at expansion factor a0, growing mode."""
    N, Np, a0 = case["N"], case["Np"], case["a0"]
    P = _params(seed)
    if a0 >= 40.0:      # a peak that is collapsing at a0
        P["delta0"] = 1.8 / a0
    m = min(N, 256)     # the linear field of a larger mesh is smooth on its scale
    dk, grid = _field(m, 1.0, P, "gauss", _normals(seed, 0, m), None)
    q, d = _displacements(m, Np, 1.0, dk, grid)
    x = torch.remainder(q + a0 * d, 1.0)
    return x, (H_I * a0 ** 1.5) * d


def _specs(case, seed):
    out, k = [], 0
    for N in MESHES:
        for _ in range(case[f"n{N}"]):
            P = _params(seed, k)
            out.append(PeakSpec(N=N, R=P["R"], delta0=P["delta0"], seed=int(seed) + k, steps=150))
            k += 1
    return out


def _kdk(N, L, q_n, x, p, schedule, gradient="spectral", smooth=0.0):
    """The KDK steps of `schedule` ((a, da) pairs) in 64 bits: yields the density after each."""
    dx = L / N
    kx, ky, kz = _kgrid(N, L)
    k2 = kx ** 2 + ky ** 2 + kz ** 2
    k2[0, 0, 0] = 1.0
    G = -1.5 * H_I ** 2 / k2
    if smooth > 0:
        G = G * torch.exp(-0.5 * k2 * (smooth * dx) ** 2)
    G[0, 0, 0] = 0.0
    del k2
    if gradient == "fd2":
        kx, ky, kz = (torch.sin(k * dx) / dx for k in (kx, ky, kz))
    elif gradient == "fd4":
        kx, ky, kz = ((8 * torch.sin(k * dx) - torch.sin(2 * k * dx)) / (6 * dx) for k in (kx, ky, kz))

    def density():
        rho = torch.zeros(N ** 3, dtype=torch.float64, device="cuda")
        for s in _parts(x.shape[0]):
            for i, w in _corners(x[s], N, dx):
                rho.index_add_(0, i, w)
        return rho.view(N, N, N) * (N ** 3 / q_n) - 1.0

    def forces(delta):      # times a
        phik = torch.fft.rfftn(delta) * G
        return [_gather(torch.fft.irfftn(-1j * kc * phik, s=(N, N, N)), x, N, dx) for kc in (kx, ky, kz)]

    def kick(acc, w):
        for c in range(3):
            p[:, c] += w * acc[c]

    def hub(a):
        return H_I * a ** -1.5

    acc = forces(density())
    for a, da in schedule:
        kick(acc, 0.5 * da / (a * hub(a)) / a)
        am = a + 0.5 * da
        for s in _parts(x.shape[0]):
            x[s] = torch.remainder(x[s] + (da / (am ** 3 * hub(am))) * p[s], L)
        delta = density()
        acc = forces(delta)
        kick(acc, 0.5 * da / ((a + da) * hub(a + da)) / (a + da))
        yield delta


def _schedule(case):
    a, out = case["a0"], []
    a_end = _a_end(case)
    for _ in range(case["steps"]):
        da = case["rate"] * a
        if case.get("schedule") == "frac":
            da = min(da, a_end - a)
        out.append((a, da))
        a += da
    return out


def _a_end(case):
    return case["a0"] * (1.0 + case["rate"]) ** (case["steps"] - 0.5)


def _snapshot(x, p, q):
    """Displacements from the lattice (nearest image) and momenta, single precision."""
    d = (x - q).to(torch.float32)
    d -= torch.round(d)
    return {"displacement": d, "momentum": p.to(torch.float32)}


TAIL = (0.02, 2.0, 10.0)


# ------------------------------------------------------------------------------ the cases
def prepare(case, seed):
    kind = case["kind"]
    if kind in ("run", "steps"):
        x, p = _particles(case, seed)
        eng = Engine([PeakConfig(N=case["N"], Np=case["Np"], L=1.0, smooth=case["smooth"], tile=case["tile"],
                                 gradient=case["gradient"])])
        return dict(case=case, engine=eng, x=x, p=p, q=_lattice(case["Np"], 1.0), schedule=_schedule(case))
    if kind == "ensemble":
        specs = _specs(case, seed)
        ens = Ensemble(specs)
        return dict(case=case, ensemble=ens, noises=[_normals(seed, k, s.N) for k, s in enumerate(specs)],
                    buffers=ens.result_buffers())
    P = _params(seed)
    st = dict(case=case, noise=_normals(seed, 0, case["N"]) if case["noise"] else None, P=P)
    if case["profile"] == "zeta":
        st["spline"] = _profile()
    return st


def run(st):
    case = st["case"]
    if case["kind"] == "run":
        eng, frac = st["engine"], case["schedule"] == "frac"
        eng.set_particles(0, st["x"], st["p"], case["a0"], mode=_lib.SCHED_FRAC if frac else _lib.SCHED_RATIO,
                          param=case["rate"], a_end=_a_end(case), max_steps=case["steps"])
        eng.run(case["steps"] + 2)      # forces at the start, the steps, the closing kick
        return dict(_snapshot(*eng.particles(0), st["q"]), delta=eng.delta(0))
    if case["kind"] == "steps":
        eng, deltas = st["engine"], []
        eng.set_particles(0, st["x"], st["p"], case["a0"])
        for a, da in st["schedule"]:
            eng.step_explicit(0, a, da)
            deltas.append(eng.delta(0))
        return dict(_snapshot(*eng.particles(0), st["q"]), delta=deltas)
    if case["kind"] == "ensemble":
        ens = st["ensemble"]
        ens.load(noises=st["noises"])
        ens.step(case["steps"] + 1)
        stats = ens.stats()
        return {"delta": ens.deltas(st["buffers"]),
                "energy": np.array([[s.kinetic, s.potential] for s in stats], dtype=np.float32)}
    P, N = st["P"], case["N"]
    if case["profile"] == "zeta":
        x, p, dl, _ = make_particles(N, case["Np"], 6.0, KIND_ZETA, P["mu"], P["axes"], spline=st["spline"],
                                     noise=st["noise"], tail_rms=TAIL[0] if case["noise"] else 0.0, tail_k=TAIL[1:],
                                     delta_lin=True)
    else:
        x, p, dl, _ = make_particles(N, case["Np"], 1.0, KIND_GAUSS, P["delta0"], P["R"], noise=st["noise"],
                                     noise_frac=0.01 if case["noise"] else 0.0, delta_lin=True)
    return {"x": x, "p": p, "delta_lin": dl}


def work(case):
    """Particle states read and written once per step, densities and force grids once per step,
    the inputs and outputs; four transforms and the CIC arithmetic per step."""
    if case["kind"] == "ensemble":
        sizes = [(N, N) for N in MESHES for _ in range(case[f"n{N}"])]
    else:
        sizes = [(case["N"], case["Np"])]
    steps = case.get("steps", 0)
    nbytes = flops = 0.0
    for N, Np in sizes:
        n, m = Np ** 3, N ** 3
        fft = 2.5 * m * math.log2(m)
        if case["kind"] != "run" and case["kind"] != "steps":       # the initial conditions
            nbytes += 8 * m * (1 if case.get("noise", True) else 0) + 48 * n
            flops += 6 * fft + 60 * n
        if case["kind"] == "ic":
            nbytes += 8 * m
            continue
        nbytes += steps * (64 * n + 16 * m)
        flops += steps * (4 * fft + 150 * n)
        nbytes += 4 * m if case["kind"] != "steps" else 4 * m * steps
        if case["kind"] != "ensemble":
            nbytes += 48 * n + 24 * n
    return {"bytes": nbytes, "flops": flops}


def exact(case, seed):
    kind = case["kind"]
    if kind in ("run", "steps"):
        x, p = _particles(case, seed)
        q = _lattice(case["Np"], 1.0)
        deltas = []
        for d in _kdk(case["N"], 1.0, case["Np"] ** 3, x, p, _schedule(case), case["gradient"], case["smooth"]):
            deltas = deltas + [d] if kind == "steps" else [d]
        d = x - q
        d -= torch.round(d)
        return {"displacement": d, "momentum": p, "delta": deltas if kind == "steps" else deltas[0]}
    if kind == "ensemble":
        out, sched = [], _schedule(dict(a0=1.0, rate=RATIO, steps=case["steps"]))
        for k, s in enumerate(_specs(case, seed)):
            P = dict(R=s.R, delta0=s.delta0)
            dk, grid = _field(s.N, 1.0, P, "gauss", _normals(seed, k, s.N), None)
            q, d = _displacements(s.N, s.N, 1.0, dk, grid)
            x, p = torch.remainder(q + d, 1.0), H_I * d
            del dk, grid, q, d
            for delta in _kdk(s.N, 1.0, s.n, x, p, sched):
                pass
            out.append(delta)
        return {"delta": out, "energy": None}
    N, Np, P = case["N"], case["Np"], _params(seed)
    L = 6.0 if case["profile"] == "zeta" else 1.0
    dk, grid = _field(N, L, P, case["profile"], _normals(seed, 0, N) if case["noise"] else None, TAIL)
    q, d = _displacements(N, Np, L, dk, grid)
    return {"x": torch.remainder(q + d, L), "p": H_I * d, "delta_lin": torch.fft.irfftn(dk, s=(N, N, N))}
