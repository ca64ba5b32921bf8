"""Workloads of the radiation calls, sized over the range they are used on.

``listed()`` names them, ``draw(rng)`` gives another of the same ranges, ``prepare(case, seed)`` sets
up what a user's program holds before the call (fields, beam, grids and the context), ``run(state)``
is one pass through the public calls, ``work(case)`` the least bytes and operations of a pass, and
``exact(case, seed)`` the same results from plain NumPy and torch in 64 bits.

The set-ups are the synthetic stand-ins of the tests and the benchmark: the 41-period planar
undulator (0.5 T, 50 mm) and the 30-period elliptical one (0.6 T / 0.4 T, 57 mm) with a 3 GeV
electron beam, batches of uneven undulator jobs, half-period tuning, and STL meshes.  The seed moves
field strengths, beam offsets, photon energies and apertures by a little, as one machine setting
differs from the next.
"""
import math
import os
import struct
import tempfile

import numpy as np
import torch

C = 2.99792458e8
H, HBAR, QE, ME = 6.62606876e-34, 1.054571596e-34, 1.602176462e-19, 9.10938356e-31
EPS0, MU0, SQRT_2PI = 8.854187817e-12, 1.2566370614e-6, 2.5066282746310002416
GAMMA_PER_GEV = QE / (1e-9 * ME * C * C)
CURRENT = 0.5
PRECISION = 0.01


def listed():
    return [
        # a scan over one harmonic's line: the shortest call, all launches and latency
        dict(name="spectrum_line", kind="spectrum", device="undulator", n=61, low=0.95, high=1.05, compute="fp64", pol="all"),
        # the usual spectrum: on axis, four harmonics, 2000 energies
        dict(name="spectrum", kind="spectrum", device="undulator", n=2000, low=0.2, high=4.4, compute="fp64", pol="all"),
        # an elliptical undulator's circularly polarised spectrum up to the ninth harmonic
        dict(name="spectrum_epu_mixed", kind="spectrum", device="epu", n=5001, low=0.5, high=9.0, compute="mixed",
             pol="circular-left"),
        # the call's default grid, one linear polarisation
        dict(name="flux_default_grid", kind="flux", device="undulator", nx=51, ny=51, width=0.01, compute="fp64",
             pol="linear-horizontal"),
        # the flux map of the benchmark, in both precisions
        dict(name="flux_map", kind="flux", device="undulator", nx=201, ny=201, width=0.01, compute="fp64", pol="all"),
        dict(name="flux_map_mixed", kind="flux", device="undulator", nx=201, ny=201, width=0.01, compute="mixed", pol="all"),
        # heat load on an absorber: the whole fan, and a smaller map of one face only
        dict(name="power_map", kind="power", device="undulator", nx=201, ny=201, width=0.03, compute="fp64", normal=0),
        dict(name="power_face_mixed", kind="power", device="epu", nx=101, ny=75, width=0.03, compute="mixed", normal=1),
        # a beam with emittance and energy spread: a new trajectory for each particle
        dict(name="flux_beam", kind="beam", device="epu", nx=51, ny=51, width=0.008, particles=16, compute="fp64"),
        # a scan of undulator designs in one call: uneven jobs, 10 to 200 periods
        dict(name="design_batch_mixed", kind="batch", jobs=32, compute="mixed"),
        # one tuning step: flux at 441 points x 256 energies and its gradient by 82 pole strengths
        dict(name="tuning_step_mixed", kind="tuning", side=21, n=256, level=12, compute="mixed"),
        # power on a meshed absorber behind a mask that shadows part of it
        dict(name="power_stl", kind="stl", side=16),
    ]


def _spread(rng, low, high):
    """A whole number between low and high, even over its logarithm."""
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(["spectrum", "spectrum", "flux", "flux", "power", "beam", "batch", "tuning", "stl"])
    device = rng.choice(["undulator", "epu"])
    compute = rng.choice(["fp64", "mixed"])
    pol = rng.choice(["all", "all", "linear-horizontal", "circular-left"])
    if kind == "spectrum":
        low = rng.uniform(0.2, 1.0)
        return dict(kind=kind, device=device, n=_spread(rng, 21, 6000), low=low, high=low + rng.uniform(0.1, 7.0),
                    compute=compute, pol=pol)
    if kind == "flux":
        return dict(kind=kind, device=device, nx=_spread(rng, 7, 201), ny=_spread(rng, 7, 201),
                    width=rng.uniform(0.002, 0.01), compute=compute, pol=pol)
    if kind == "power":
        return dict(kind=kind, device=device, nx=_spread(rng, 7, 201), ny=_spread(rng, 7, 201),
                    width=rng.uniform(0.01, 0.04), compute=compute, normal=rng.choice([0, 1]))
    if kind == "beam":
        return dict(kind=kind, device=device, nx=_spread(rng, 5, 51), ny=_spread(rng, 5, 51),
                    width=rng.uniform(0.002, 0.008), particles=_spread(rng, 3, 16), compute="fp64")
    if kind == "batch":
        return dict(kind=kind, jobs=_spread(rng, 3, 20), compute="mixed")
    if kind == "tuning":
        return dict(kind=kind, side=rng.randint(3, 21), n=_spread(rng, 9, 256), level=rng.randint(10, 12), compute=compute)
    return dict(kind=kind, side=rng.randint(3, 16))


# ---- one machine setting: plain numbers from the case and the seed ----------------------------------
def _first_harmonic(bx, by, period, gev):
    """Photon energy [eV] of the first harmonic on axis, from K of both field components."""
    k2 = sum((QE * b * period / (2 * math.pi * ME * C)) ** 2 for b in (bx, by))
    g = gev * GAMMA_PER_GEV
    return H * C / QE / (period / (2 * g * g) * (1 + k2 / 2))


def _setting(case, seed):
    r = np.random.default_rng(seed)
    s = {"gev": 3.0 * (1 + 1e-4 * r.standard_normal()), "span": (-1.5, 1.5),
         "x0": [float(v) for v in 20e-6 * r.standard_normal(2)] + [0.0], "obs": [0.0, 0.0, 30.0 + 0.05 * r.standard_normal()]}
    if case.get("device") == "epu":
        by, bx = 0.6 * (1 + 2e-3 * r.standard_normal()), 0.4 * (1 + 2e-3 * r.standard_normal())
        s["fields"] = [dict(bfield=[0.0, by, 0.0], period=0.057, n=30, phase=-math.pi / 2, scale=None),
                       dict(bfield=[bx, 0.0, 0.0], period=0.057, n=30, phase=0.0, scale=None)]
        s["points"], s["e1"], s["periods"] = 16001, _first_harmonic(bx, by, 0.057, s["gev"]), 30
    else:
        by = 0.5 * (1 + 2e-3 * r.standard_normal())
        s["fields"] = [dict(bfield=[0.0, by, 0.0], period=0.05, n=41, phase=-math.pi / 2, scale=None)]
        s["points"], s["e1"], s["periods"] = 20001, _first_harmonic(0.0, by, 0.05, s["gev"]), 41
    s["size"] = 1 + 0.02 * r.standard_normal()
    return s, r


def _beam(s):
    return dict(type="electron", energy_GeV=s["gev"], x0=s["x0"], d0=[0, 0, 1], current=CURRENT)


def _machine(s):
    from oscars_b200.sr import sr
    o = sr(gpu=1)
    for f in s["fields"]:
        o.add_bfield_undulator(bfield=f["bfield"], period=[0, 0, f["period"]], nperiods=f["n"], phase=f["phase"])
    o.set_particle_beam(**_beam(s))
    o.set_ctstartstop(*s["span"])
    o.set_npoints_trajectory(s["points"])
    return o


def _energies(case, s):
    return np.linspace(case["low"] * s["e1"], case["high"] * s["e1"], case["n"])


def _jobs(case, seed):
    """Undulator designs: 15-100 mm, 0.2-1.2 T, 10-200 periods, 1-4096 observers x 1-256 energies."""
    r = np.random.default_rng(seed)
    jobs = []
    shape = np.random.default_rng(case["jobs"])  # the sizes are the case's, the strengths the seed's
    for _ in range(case["jobs"]):
        lam, b, n = shape.uniform(0.015, 0.1), shape.uniform(0.2, 1.2) * (1 + 1e-3 * r.standard_normal()), int(shape.integers(10, 201))
        half = lam * (n + 2) / 2 + 0.2
        nx, ny, ne = int(shape.integers(1, 65)), int(shape.integers(1, 65)), int(shape.integers(1, 257))
        wx, wy = shape.uniform(0.001, 0.006, 2) * (1 + 1e-2 * r.standard_normal())
        z = shape.uniform(20, 40)
        x = np.linspace(-wx / 2, wx / 2, nx) if nx > 1 else np.zeros(1)
        y = np.linspace(-wy / 2, wy / 2, ny) if ny > 1 else np.zeros(1)
        X, Y = np.meshgrid(x, y, indexing="ij")
        e1 = _first_harmonic(0.0, b, lam, 3.0)
        jobs.append({"gev": 3.0, "span": (-half, half), "x0": [0.0, 0.0, 0.0], "points": int(np.clip(240 * (n + 2 + 0.4 / lam), 4096, 65536)),
                     "fields": [dict(bfield=[0.0, b, 0.0], period=lam, n=n, phase=-math.pi / 2, scale=None)], "periods": n,
                     "obs": np.stack([X.ravel(), Y.ravel(), np.full(X.size, z)], 1), "energies": np.linspace(0.95 * e1, 1.05 * e1, ne)})
    return jobs


def _tuning(case, seed):
    r = np.random.default_rng(seed)
    x = np.linspace(-0.001, 0.001, case["side"]) * (1 + 1e-2 * r.standard_normal())
    X, Y = np.meshgrid(x, x, indexing="ij")
    e1 = _first_harmonic(0.0, 0.5, 0.05, 3.0)
    return (np.stack([X.ravel(), Y.ravel(), np.full(X.size, 30.0)], 1), np.linspace(0.95 * e1, 1.05 * e1, case["n"]),
            [1 + 0.005 * r.standard_normal(82) for _ in range(2)])


def _mesh(case, seed):
    """A flat absorber of side x side squares at 20 m and a two-triangle mask at 10 m: facets as
    float32 vertices (n, 3, 3), the mask's in millimetres."""
    r = np.random.default_rng(seed + 1)
    n, w = case["side"], 0.02 * (1 + 0.02 * r.standard_normal())
    g = np.linspace(-w / 2, w / 2, n + 1)
    plate = []
    for i in range(n):
        for j in range(n):
            p = [(g[i], g[j], 0.0), (g[i + 1], g[j], 0.0), (g[i + 1], g[j + 1], 0.0), (g[i], g[j + 1], 0.0)]
            plate += [[p[0], p[1], p[2]], [p[0], p[2], p[3]]]
    h = 3.3 * (1 + 0.02 * r.standard_normal())
    q = [(-3.0, 0.0, 0.0), (3.0, 0.0, 0.0), (3.0, h, 0.0), (-3.0, h, 0.0)]
    return np.array(plate, np.float32), np.array([[q[0], q[1], q[2]], [q[0], q[2], q[3]]], np.float32)


def _write_mesh(tri, nz):
    f = tempfile.NamedTemporaryFile(suffix=".stl", delete=False)
    with f:
        f.write(b"mesh".ljust(80, b"\0") + struct.pack("<I", len(tri)))
        for t in tri:
            f.write(struct.pack("<12fH", 0.0, 0.0, nz, *t.ravel().tolist(), 0))
    return f.name


# ---- what a program holds, and one pass -----------------------------------------------------------
def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        from oscars_b200.batch import BatchRunner, Job, undulator
        jobs = [Job(fields=[undulator(f["bfield"], [0, 0, f["period"]], f["n"], phase=f["phase"]) for f in j["fields"]], energy_GeV=j["gev"],
                    ctstartstop=j["span"], npoints=j["points"], obs=j["obs"], energies_eV=j["energies"], current=CURRENT)
                for j in _jobs(case, seed)]
        return dict(kind=kind, case=case, runner=BatchRunner(gpu=0), jobs=jobs)
    if kind == "tuning":
        from oscars_b200.tuning import TuningProblem
        obs, energies, factors = _tuning(case, seed)
        p = TuningProblem(bfield=[0, 0.5, 0], period=[0, 0, 0.05], nperiods=41, obs=obs, energies_eV=energies, level=case["level"],
                          compute=case["compute"])
        return dict(kind=kind, case=case, problem=p, target=torch.from_numpy(p.flux(np.ones(82))), factors=[torch.from_numpy(f) for f in factors], step=0)
    s, _ = _setting(case, seed)
    o = _machine(s)
    state = dict(kind=kind, case=case, sr=o, s=s, seed=seed % 100000 + 1)
    if kind == "spectrum":
        state["energies"] = _energies(case, s).tolist()
    elif kind == "beam":
        o.set_particle_beam(**_beam(s), sigma_energy_GeV=0.003, beta=[1.5, 0.8], alpha=[0, 0], emittance=[0.9e-9, 8e-12])
    elif kind == "stl":
        plate, mask = _mesh(case, seed)
        for tri, nz, scale, z in ((plate, 1.0, 1, 20.0), (mask, -1.0, 0.001, 10.0)):
            path = _write_mesh(tri, nz)
            o.add_stl(path, scale=scale, translation=[0, 0, z])
            os.unlink(path)
    return state


def run(state):
    case, kind = state["case"], state["kind"]
    if kind == "batch":
        return {"flux": state["runner"].flux(state["jobs"], compute=case["compute"])}
    if kind == "tuning":
        from oscars_b200.tuning import UndulatorFlux
        f = state["factors"][state["step"] % 2].clone().requires_grad_()  # new pole strengths at every step
        state["step"] += 1
        flux = UndulatorFlux.apply(f, state["problem"])
        ((flux - state["target"]) ** 2).sum().backward()
        return {"flux": flux, "gradient": f.grad}
    o, s = state["sr"], state["s"]
    if kind == "spectrum":
        e, v = o.calculate_spectrum(obs=s["obs"], energy_points_eV=state["energies"], polarization=case["pol"], compute=case["compute"],
                                    return_numpy=True)
        return {"points": e, "values": v, "levels": o.last_levels}
    if kind == "stl":
        r = o.calculate_power_density_stl(farfield_origin=[0, 0, 0])
        return {"values": np.array([p for _, p in r]), "levels": o.last_levels}
    w = case["width"] * s["size"]
    grid = dict(npoints=[case["nx"], case["ny"]], plane="XY", width=[w, w], translation=s["obs"], return_numpy=True)
    if kind == "power":
        x, v = o.calculate_power_density_rectangle(normal=case["normal"], compute=case["compute"], **grid)
    elif kind == "beam":
        o.set_seed(state["seed"])
        x, v = o.calculate_flux_rectangle(energy_eV=s["e1"], nparticles=case["particles"], compute=case["compute"], **grid)
    else:
        x, v = o.calculate_flux_rectangle(energy_eV=s["e1"], polarization=case["pol"], compute=case["compute"], **grid)
    return {"points": x, "values": v, "levels": o.last_levels}


# ---- least work -------------------------------------------------------------------------------------
def _ladder(periods, harmonic):
    """Samples of the levels a converged entry needs: level 9 at least, two samples per cycle."""
    level = max(9, math.ceil(math.log2(2.5 * periods * harmonic)))
    return 2 ** (level + 1) - 1


def work(case):
    # an observer's amplitude at one sample takes about 55 operations, an energy's phase, sine, cosine
    # and sums about 35, power density 60, a ray against a mesh that does not shadow it 20
    kind = case["kind"]
    if kind == "batch":
        flops = nbytes = 0
        for j in _jobs(case, 0):
            p, e = len(j["obs"]), len(j["energies"])
            flops += p * _ladder(j["periods"], 1) * (55 + 35 * e) + 350 * j["points"]
            nbytes += 8 * (3 * p + e + p * e)
        return {"bytes": nbytes, "flops": flops}
    if kind == "tuning":
        p, e = case["side"] ** 2, case["n"]
        return {"bytes": 8 * (3 * p + e + 3 * p * e), "flops": 3 * p * (2 ** (case["level"] + 1) - 1) * (55 + 35 * e) + 3 * 350 * 20001}
    s, _ = _setting(case, 0)
    if kind == "spectrum":
        return {"bytes": 16 * case["n"], "flops": _ladder(s["periods"], case["high"]) * (55 + 35 * case["n"])}
    if kind == "stl":
        n = 2 * case["side"] ** 2 + 2
        return {"bytes": 8 * 16 * n, "flops": n * _ladder(s["periods"], 1) * 80}
    p = case["nx"] * case["ny"]
    if kind == "power":
        return {"bytes": 8 * 4 * p, "flops": p * _ladder(s["periods"], 1) * 60}
    q = case.get("particles", 1)
    return {"bytes": 8 * 4 * p, "flops": q * (p * _ladder(s["periods"], 1) * 90 + 350 * s["points"])}


# ---- the same results in 64 bits ----------------------------------------------------------------------
def _trajectories(settings):
    """Per setting (t, y (9, n), y'' (9, n), gamma): classical RK4 from the start point in both
    directions, all settings and directions as lanes of one array, and the clamped spline through the
    points.  The acceleration stored with a point is the previous one's, as the calls define it."""
    lanes = [(k, d) for k in range(len(settings)) for d in (1, -1)]
    nf = max(len(s["fields"]) for s in settings)
    amp, per, cnt, shift = np.zeros((nf, 2, len(lanes))), np.ones((nf, len(lanes))), np.zeros((nf, len(lanes))), np.zeros((nf, len(lanes)))
    half = [None] * nf
    h, steps, x = np.zeros(len(lanes)), np.zeros(len(lanes), int), np.zeros((6, len(lanes)))
    qomg = np.zeros(len(lanes))
    for i, (k, d) in enumerate(lanes):
        s = settings[k]
        g = s["gev"] * GAMMA_PER_GEV
        b = math.sqrt(1.0 - 1.0 / (g * g))
        g = 1.0 / math.sqrt(1.0 - b * b)
        dt = (s["span"][1] - s["span"][0]) / C / (s["points"] - 1)
        h[i] = d * dt
        steps[i] = int(1 + s["span"][1] / C / dt) if d > 0 else int(-s["span"][0] / C / dt)
        x[:, i] = [s["x0"][0], 0.0, s["x0"][1], 0.0, s["x0"][2], b * C]
        qomg[i] = -QE / ME / g
        for j, f in enumerate(s["fields"]):
            amp[j, :, i], per[j, i], cnt[j, i] = f["bfield"][:2], f["period"], f["n"]
            shift[j, i] = f["phase"] * f["period"] / (2 * math.pi)
            if f["scale"] is not None:
                half[j] = np.asarray(f["scale"])
    length = per * (cnt + 2)

    def field(z):
        b = np.zeros((2, len(lanes)))
        for j in range(nf):
            u = z - shift[j]
            a = np.abs(u)
            e = length[j] / 2 - a  # distance to the nearer end: quarter, three-quarter, then full poles
            w = np.where(e < 0, 0.0, np.where(e < per[j] / 2, 0.25, np.where(e < per[j], 0.75, 1.0)))
            if half[j] is not None:
                k = np.clip(((u + length[j] / 2 - per[j]) / (per[j] / 2)).astype(int), 0, len(half[j]) - 1)
                w = np.where(w == 1.0, half[j][k], w)
            b += amp[j] * (w * np.sin(2 * math.pi * u / per[j]))
        return b

    def slope(v):
        b = field(v[4])
        return np.stack([v[1], qomg * (-v[5] * b[1]), v[3], qomg * (v[5] * b[0]), v[5], qomg * (v[1] * b[1] - v[3] * b[0])])

    top = int(steps.max()) + 1
    at, acc = np.zeros((top, 6, len(lanes))), np.zeros((top, 3, len(lanes)))
    k1 = slope(x)
    at[0], acc[0] = x, k1[1::2]
    for i in range(1, top):
        acc[i] = k1[1::2]
        k2 = slope(x + 0.5 * h * k1)
        k3 = slope(x + 0.5 * h * k2)
        k4 = slope(x + h * k3)
        x = x + h / 6.0 * (k1 + k4 + 2.0 * (k2 + k3))
        at[i] = x
        k1 = slope(x)
    out = []
    for k, s in enumerate(settings):
        fw, bw = 2 * k, 2 * k + 1
        nfw, nbw = steps[fw], steps[bw]
        order = lambda v: np.concatenate([v[1:nbw + 1, :, bw][::-1], v[:nfw, :, fw]])  # noqa: E731
        a, c = order(at), order(acc)
        t = np.concatenate([h[bw] * np.arange(1, nbw + 1)[::-1], h[fw] * np.arange(nfw)])
        y = np.concatenate([a[:, ::2].T, a[:, 1::2].T / C, c.T / C])
        out.append((t, y, _spline(t, y), -QE / ME / qomg[fw]))
    return out


def _spline(t, y):
    n = len(t)
    d, out, u = np.zeros(n), np.zeros((n, 9)), np.zeros((n, 9))
    yt = y.T
    first, step = np.diff(t), np.diff(yt, axis=0) / np.diff(t)[:, None]
    d[0] = -0.5
    sig = (t[1:-1] - t[:-2]) / (t[2:] - t[:-2])
    right = 6.0 * (step[1:] - step[:-1]) / (t[2:] - t[:-2])[:, None]
    del first
    for i in range(1, n - 1):
        p = sig[i - 1] * d[i - 1] + 2.0
        d[i] = (sig[i - 1] - 1.0) / p
        u[i] = (right[i - 1] - sig[i - 1] * u[i - 1]) / p
    out[-1] = -0.5 * u[n - 2] / (0.5 * d[n - 2] + 1.0)
    for i in range(n - 2, -1, -1):
        out[i] = d[i] * out[i + 1] + u[i]
    return out.T.copy()


def _samples(track, level):
    """The 2^level samples of one level as tensors: t, and the nine components."""
    t, y, ypp, _ = track
    n = 2 ** level
    T = t[0] + (t[-1] - t[0]) / 2 ** (level + 1) + (t[-1] - t[0]) / n * np.arange(n)
    k = np.clip(np.searchsorted(t, T, side="right") - 1, 0, len(t) - 2)
    w = t[k + 1] - t[k]
    a, b = (t[k + 1] - T) / w, (T - t[k]) / w
    v = a * y[:, k] + b * y[:, k + 1] + ((a ** 3 - a) * ypp[:, k] + (b ** 3 - b) * ypp[:, k + 1]) * (w * w) / 6.0
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    return torch.from_numpy(T).to(dev), torch.from_numpy(v).to(dev)


def _step(track, level):
    return (track[0][-1] - track[0][0]) / (2.0 ** (level + 1) - 1)


def _wave(smp, obs, omega):
    """Complex sums (entries, 3) over the samples and the largest phase step, entry by entry."""
    T, v = smp
    R = [obs[:, c, None] - v[c] for c in range(3)]
    D = torch.sqrt(R[0] * R[0] + R[1] * R[1] + R[2] * R[2])
    ph = -omega[:, None] * (T + D / C)
    n = [r / D for r in R]
    b, a = v[3:6], v[6:9]
    om = 1.0 - (n[0] * b[0] + n[1] * b[1] + n[2] * b[2])
    u = [n[c] - b[c] for c in range(3)]
    near = (1.0 - (b[0] * b[0] + b[1] * b[1] + b[2] * b[2])) / (D * D * om * om)
    far = 1.0 / (D * om * om)
    w = [u[1] * a[2] - u[2] * a[1], u[2] * a[0] - u[0] * a[2], u[0] * a[1] - u[1] * a[0]]
    x = [n[1] * w[2] - n[2] * w[1], n[2] * w[0] - n[0] * w[2], n[0] * w[1] - n[1] * w[0]]
    e = torch.polar(torch.ones_like(ph), ph)
    S = torch.stack([((u[c] * near + x[c] * far) * e).sum(1) for c in range(3)], 1)
    step = (ph[:, 1:] - ph[:, :-1]).abs().amax(1) if ph.shape[1] > 1 else torch.zeros_like(omega)
    return S, step


def _polarisation(name):
    k = math.sqrt(0.5)
    return {"all": None, "linear-horizontal": [1, 0, 0], "circular-left": [k, 1j * k, 0]}[name]


def _radiation(track, obs, energies, pol="all", level=None):
    """Flux and the level it stopped at of every (observer, energy) entry."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    q = QE
    c0, c2 = q / (4 * math.pi * C * EPS0 * SQRT_2PI), 4 * math.pi * CURRENT / (H * q * MU0 * C) * 1e-6 * 0.001
    O = torch.tensor(np.asarray(obs, float), device=dev).repeat_interleave(len(energies), 0)
    W = torch.tensor(np.asarray(energies) * QE / HBAR, device=dev).repeat(len(obs))
    P = _polarisation(pol)
    P = None if P is None else torch.tensor(P, dtype=torch.complex128, device=dev)
    N = len(W)
    S, last, flux = torch.zeros(N, 3, dtype=torch.complex128, device=dev), torch.full((N,), -1.0, dtype=torch.float64, device=dev), torch.zeros(N, dtype=torch.float64, device=dev)
    at, live = torch.full((N,), -1, dtype=torch.int32, device=dev), torch.arange(N, device=dev)

    def square(s):
        if P is not None:
            s = (s * P).sum(1, keepdim=True) * P
        return (s.real ** 2 + s.imag ** 2).sum(1)

    for L in range(level + 1 if level is not None else 21):
        smp, dt = _samples(track, L), _step(track, L)
        steps = []
        part = max(1, 2 ** 23 // 2 ** L)
        for i in range(0, len(live), part):
            k = live[i:i + part]
            s, d = _wave(smp, O[k], W[k])
            S[k] += s
            steps.append(d)
        this = square(S[live] * dt)
        stop = (((this - last[live]).abs() / last[live] < PRECISION) & (torch.cat(steps) < math.pi)) if L > 8 and level is None else torch.zeros_like(this, dtype=torch.bool)
        if level is not None and L == level:
            stop = ~stop
        done = live[stop]
        flux[done] = c2 * square(S[done] * (c0 * dt))
        at[done] = L
        last[live] = this
        live = live[~stop]
        if not len(live):
            break
    return flux.cpu().numpy(), at.cpu().numpy()


def _power(smp, obs, nrm, one_sided):
    T, v = smp
    R = [obs[:, c, None] - v[c] for c in range(3)]
    D2 = R[0] * R[0] + R[1] * R[1] + R[2] * R[2]
    D = torch.sqrt(D2)
    n = [r / D for r in R]
    b, a = v[3:6], v[6:9]
    u = [n[c] - b[c] for c in range(3)]
    w = [u[1] * a[2] - u[2] * a[1], u[2] * a[0] - u[0] * a[2], u[0] * a[1] - u[1] * a[0]]
    x = [n[1] * w[2] - n[2] * w[1], n[2] * w[0] - n[0] * w[2], n[0] * w[1] - n[1] * w[0]]
    om = 1.0 - (b[0] * n[0] + b[1] * n[1] + b[2] * n[2])
    face = 1.0 if nrm is None else n[0] * nrm[0] + n[1] * nrm[1] + n[2] * nrm[2]
    t = (x[0] ** 2 + x[1] ** 2 + x[2] ** 2) / om ** 5 / D2 * face
    return torch.where(face > 0, t, torch.zeros_like(t)) if one_sided else t


def _power_density(track, obs, normal):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    O = torch.tensor(np.asarray(obs, float), device=dev)
    nrm = (0.0, 0.0, 1.0)
    N = len(O)
    S, last, out = (torch.full((N,), v, dtype=torch.float64, device=dev) for v in (0.0, -1.0, 0.0))
    at, live = torch.full((N,), -1, dtype=torch.int32, device=dev), torch.arange(N, device=dev)
    scale = QE * CURRENT / (16 * math.pi ** 2 * EPS0 * C) / 1e6
    for L in range(21):
        smp, dt = _samples(track, L), _step(track, L)
        part = max(1, 2 ** 23 // 2 ** L)
        for i in range(0, len(live), part):
            k = live[i:i + part]
            S[k] += _power(smp, O[k], nrm if normal else None, bool(normal)).sum(1)
        B = smp[1][3:6]
        turn = float((B[:, 1:] - B[:, :-1]).square().sum(0).sqrt().max()) if L else 0.0
        this = S[live] * dt
        stop = ((this - last[live]).abs() / last[live] < PRECISION) | (this == last[live]) if L > 8 and turn < 2 / track[3] else torch.zeros_like(this, dtype=torch.bool)
        if L > 8 and turn >= 2 / track[3]:
            stop = this == last[live]
        done = live[stop]
        out[done] = S[done] * (scale * dt)
        at[done] = L
        last[live] = this
        live = live[~stop]
        if not len(live):
            break
    return out.cpu().numpy(), at.cpu().numpy()


def _blocked(origin, target, tri, self_index):
    """Whether another facet lies between each sample and the facet's centre (Moller-Trumbore)."""
    to = target - origin
    dist = to.square().sum(1).sqrt()
    d = to / dist[:, None]
    A, e1, e2 = tri[:, 0], tri[:, 1] - tri[:, 0], tri[:, 2] - tri[:, 0]
    cross = lambda p, q: torch.stack([p[..., 1] * q[..., 2] - p[..., 2] * q[..., 1], p[..., 2] * q[..., 0] - p[..., 0] * q[..., 2], p[..., 0] * q[..., 1] - p[..., 1] * q[..., 0]], -1)  # noqa: E731
    p = cross(d[:, None], e2[None])
    det = (e1[None] * p).sum(-1)
    s = origin[:, None] - A[None]
    u = (s * p).sum(-1) / det
    q = cross(s, e1[None])
    v = (d[:, None] * q).sum(-1) / det
    t = (e2[None] * q).sum(-1) / det
    hit = (det.abs() >= 1e-12) & (u >= 0) & (u <= 1) & (v >= 0) & (u + v <= 1) & (t > 0) & (t < dist[:, None])
    hit[:, self_index] = False
    return hit.any(1)


def _power_mesh(track, tri, nrm):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    centre = torch.tensor(((tri[:, 0] + tri[:, 1]) + tri[:, 2]) / 3.0, device=dev)
    tri = torch.tensor(tri, device=dev)
    n = len(tri)
    S, last, out, at, live = np.zeros(n), -np.ones(n), np.zeros(n), -np.ones(n, np.int32), list(range(n))
    scale = QE * CURRENT / (16 * math.pi ** 2 * EPS0 * C) / 1e6
    for L in range(15):
        smp, dt = _samples(track, L), _step(track, L)
        X, B = smp[1][0:3].T.contiguous(), smp[1][3:6].T.contiguous()
        rest = []
        for i in live:
            seen = ~_blocked(X, centre[i], tri, i)
            S[i] += float((_power(smp, centre[i][None], nrm[i], False)[0].abs() * seen).sum())
            k = torch.nonzero(seen).ravel()
            before = torch.cat([torch.zeros(1, 3, dtype=B.dtype, device=dev), B[k][:-1]])
            turn = (B[k] - before).square().sum(1).sqrt()[k > 0]
            turn = float(turn.max()) if len(turn) else -1.0
            this = S[i] * dt
            with np.errstate(all="ignore"):
                near = abs(this - last[i]) / last[i] < PRECISION
            if L > 8 and ((near and turn < 2 / track[3]) or this == last[i]):
                at[i] = L
            else:
                rest.append(i)
            out[i], last[i] = S[i] * (scale * dt), this
        live = rest
        if not live:
            break
    return out, np.maximum.accumulate(at) if (at < 0).any() else at


def exact(case, seed):
    kind = case["kind"]
    if kind == "beam":
        return None  # the particles are drawn by the call itself
    if kind == "batch":
        jobs = _jobs(case, seed)
        return {"flux": [_radiation(t, j["obs"], j["energies"])[0].reshape(len(j["obs"]), -1) for t, j in zip(_trajectories(jobs), jobs)]}
    if kind == "tuning":
        obs, energies, factors = _tuning(case, seed)
        s = {"gev": 3.0, "span": (-1.5, 1.5), "x0": [0.0, 0.0, 0.0], "points": 20001,
             "fields": [dict(bfield=[0.0, 0.5, 0.0], period=0.05, n=41, phase=-math.pi / 2, scale=factors[0])]}
        flux = _radiation(_trajectories([s])[0], obs, energies, level=case["level"])[0]
        return {"flux": flux.reshape(len(obs), -1), "gradient": None}  # (reverse mode through 20001 steps)
    s, _ = _setting(case, seed)
    track = _trajectories([s])[0]
    if kind == "spectrum":
        e = _energies(case, s)
        v, at = _radiation(track, [s["obs"]], e, case["pol"])
        return {"points": e, "values": v, "levels": at}
    if kind == "stl":
        plate, mask = _mesh(case, seed)
        tri = np.concatenate([plate.astype(float) + [0, 0, 20.0], mask.astype(float) * 0.001 + [0, 0, 10.0]])
        v, at = _power_mesh(track, tri, [(0.0, 0.0, 1.0)] * len(plate) + [(0.0, 0.0, -1.0)] * len(mask))
        return {"values": v, "levels": at}
    w, nx, ny = case["width"] * s["size"], case["nx"], case["ny"]
    i, j = np.divmod(np.arange(nx * ny), ny)
    d1, d2 = w / (nx - 1), w / (ny - 1)
    obs = np.stack([(-w / 2 + s["obs"][0]) + d1 * i, (-w / 2 + s["obs"][1]) + d2 * j, np.full(nx * ny, s["obs"][2])], 1)
    points = np.stack([d1 * i - d1 * (nx - 1) / 2, d2 * j - d2 * (ny - 1) / 2, np.zeros(nx * ny)], 1)
    v, at = _power_density(track, obs, case["normal"]) if kind == "power" else _radiation(track, obs, [s["e1"]], case["pol"])
    return {"points": points, "values": v, "levels": at}
