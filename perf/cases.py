"""What the solver's users have it do, as timed cases.

A case is one call (or one segment of steps) through the package's public entry
points: whole plain runs from the 40 um chamber to the 5 um columns,
the float64 validation run, segments of the grids that stream from HBM up to
the 5 um full electrode, gradients of k_s, and batched sweeps. Sizes are those
of the benchmark, the test configurations and the 10 um ladder, and odd ones
between them.

Runs with float32 fields are compared in float32: the record a Result keeps is
held in float64 arrays, but its values were computed in float32 fields.
"""

from __future__ import annotations

import importlib
import math
import random
import warnings

import numpy as np
import torch

PACKAGE = "iontracks-pulsedproton-python_gb300"
ALPHA = 1.60e-6  # volume recombination coefficient, cm^3/s
LET_KEV_UM, TRACK_RADIUS_CM = 0.0011994843758452705, 0.002  # protons of 56.2 MeV/u in air
TWO_SPECIES = dict(mu_positive_cm2_Vs=1.36, mu_negative_cm2_Vs=2.10, D_positive_cm2_s=2.82e-2, D_negative_cm2_s=4.35e-2)
L2_BYTES = 126_000_000


def _chamber(um, radius_cm, **kw):
    c = dict(um=um, radius_cm=radius_cm, volts=300.0, gap_cm=0.2, dose=8.91, pulse_us=540.0, pulses=1,
             wall="absorbing", two_species=False, dtype="float32")
    c.update(kw)
    return c


def listed():
    return [
        # the 40 um chamber of the quick checks: a few hundred tiny steps, the call's own latency
        dict(name="run_tiny", kind="run", **_chamber(40.0, 0.004)),
        # a pulse train of a 40 um chamber: nearly all of its steps are idle ones
        dict(name="run_train", kind="run", **_chamber(40.0, 0.006, pulses=3, wall="reflecting")),
        # the benchmark's 10 um column, absorbing wall (the default)
        dict(name="run_column_24", kind="run", **_chamber(10.0, 0.008)),
        # a 5 um column of odd width, two carrier species, reflecting wall, as the AIC-144 studies run it
        dict(name="run_column_59", kind="run", **_chamber(5.0, 0.0127, wall="reflecting", two_species=True)),
        # the validation run in float64 of a row of the 10 um ladder
        dict(name="run_f64", kind="run", **_chamber(10.0, 0.014, wall="reflecting", two_species=True, dtype="float64")),
        # the start of a 5 um column that no longer fits the L2, through the whole driver
        dict(name="run_start_208", kind="run", max_steps=256, **_chamber(5.0, 0.05)),
        # steps of a mid-sized 5 um column, part depositing, part idle
        dict(name="segment_330", kind="segment", pulse_steps=12, idle_steps=4, **_chamber(5.0, 0.0805)),
        # steps of the 5 um full electrode, the headline workload
        dict(name="segment_1068", kind="segment", pulse_steps=6, idle_steps=2, **_chamber(5.0, 0.265)),
        # k_s and its gradient on the 10 um column that alpha and mobility fits use
        dict(name="gradient_48", kind="gradient", checkpoint_every=64, **_chamber(10.0, 0.02)),
        # the gradient of the start of a 5 um column (reverse steps that stream from HBM)
        dict(name="gradient_208", kind="gradient", max_steps=96, checkpoint_every=32,
             **_chamber(5.0, 0.05, wall="reflecting")),
        # a small saturation curve
        dict(name="batch_8", kind="batch", configs=8, meta=5, dose=8.91, dtype="float32"),
        # the larger saturation sweep
        dict(name="batch_32", kind="batch", configs=32, meta=20260527, dose=8.91, dtype="float32"),
    ]


def draw(rng: random.Random):
    kind = rng.choice(["run", "run", "run", "segment", "segment", "gradient", "batch"])
    log = lambda a, b: math.exp(rng.uniform(math.log(a), math.log(b)))  # noqa: E731
    if kind == "batch":
        return dict(kind=kind, configs=int(round(log(4, 28))), meta=rng.randrange(1, 1000), dose=round(log(2.0, 9.0), 3),
                    dtype="float32")
    common = dict(volts=round(log(150.0, 400.0), 1), dose=round(log(1.0, 10.0), 3),
                  pulse_us=round(rng.uniform(300.0, 800.0), 1), wall=rng.choice(["absorbing", "reflecting"]),
                  two_species=rng.random() < 0.5)
    if kind == "run":
        um = rng.choice([5.0, 10.0, 10.0, 40.0])
        half = {5.0: log(8, 34), 10.0: log(4, 48), 40.0: log(1, 20)}[um]
        f64 = um != 5.0 and half < 16 and rng.random() < 0.25
        return dict(kind=kind, **_chamber(um, round(half * um * 1e-4, 6), gap_cm=rng.choice([0.1, 0.2]),
                                          dtype="float64" if f64 else "float32", **common))
    if kind == "segment":
        um = rng.choice([5.0, 10.0])
        half = log(75, 530)
        steps = 2 * rng.randrange(2, 9)
        idle = rng.randrange(0, steps)
        return dict(kind=kind, pulse_steps=steps - idle, idle_steps=idle,
                    **_chamber(um, round(half * um * 1e-4, 6), gap_cm=rng.choice([0.1, 0.2]), **common))
    if rng.random() < 0.5:
        return dict(kind=kind, checkpoint_every=rng.choice([16, 50, 64]),
                    **_chamber(10.0, round(log(4, 24) * 1e-3, 6), gap_cm=rng.choice([0.1, 0.2]), **common))
    steps = rng.randrange(20, 97)
    return dict(kind=kind, max_steps=steps, checkpoint_every=rng.choice([16, 32]),
                **_chamber(5.0, round(log(30, 150) * 5e-4, 6), **common))


# --- a user's objects -------------------------------------------------------


def _kwargs(case, seed):
    kw = dict(E_MeV_u=56.2, voltage_V=case["volts"], electrode_gap_cm=case["gap_cm"], dose_rate_Gy_s=case["dose"],
              pulse_duration_s=case["pulse_us"] * 1e-6, repetition_rate_hz=50.0, n_pulses=case["pulses"],
              grid_size_um=case["um"], sampled_radius_cm=case["radius_cm"], lateral_boundary=case["wall"],
              max_voxels=2e9, seed=int(seed))
    if case["two_species"]:
        kw.update(TWO_SPECIES)
    return kw


def _sweep_kwargs(case, seed):
    """Voltages over 100-400 V, the other ranges those of the 64-grid saturation sweep."""
    r = np.random.default_rng(case["meta"])
    out = []
    for i, volts in enumerate(np.logspace(np.log10(100.0), np.log10(400.0), case["configs"])):
        um = float(r.choice([5.0, 10.0]))
        gap = float(r.choice([0.1, 0.2, 0.3]))
        out.append(dict(E_MeV_u=56.2, voltage_V=float(volts), electrode_gap_cm=gap, dose_rate_Gy_s=case["dose"],
                        pulse_duration_s=float(r.uniform(100e-6, 1000e-6)), repetition_rate_hz=50.0, n_pulses=1,
                        grid_size_um=um, sampled_radius_cm=float(r.uniform(0.008, 0.03)),
                        lateral_boundary="absorbing", max_voxels=2e9, seed=int(seed) * 1000 + i))
    return out


def _package():
    return importlib.import_module(PACKAGE)


def _config(kw):
    with warnings.catch_warnings():
        warnings.simplefilter("ignore")
        return _package().SimulationConfig(**kw)


def prepare(case, seed):
    kind = case["kind"]
    state = dict(case=case)
    if kind == "batch":
        state["configs"] = [_config(kw) for kw in _sweep_kwargs(case, seed)]
    else:
        state["config"] = _config(_kwargs(case, seed))
    if kind == "segment":
        engine = importlib.import_module(PACKAGE + ".engine")
        s = _scalars(_kwargs(case, seed))
        offsets, xs, ys = _segment_tracks(case, s, seed)
        eng = engine.ChamberEngine(state["config"], dtype=case["dtype"], max_tracks=max(1, len(xs)),
                                   tally_steps=len(offsets) - 1)
        eng.upload_tracks(xs, ys)
        for k, f in enumerate((eng.pos[0], eng.neg[0])):
            _fill(f[:, :, : s["nzb"]], s, 2 * int(seed) + k)
        state.update(engine=eng, offsets=offsets)
    return state


def run(state):
    case, kind, pkg = state["case"], state["case"]["kind"], _package()
    if kind == "run":
        fields = _wants_fields(case)
        r = pkg.run_simulation_b200(state["config"], progress=False, dtype=case["dtype"],
                                    max_steps=case.get("max_steps"), return_fields=fields)
        return _record([r], case["dtype"], ks="max_steps" not in case, fields=fields)
    if kind == "segment":
        eng = state["engine"]
        eng.run_segment(state["offsets"], tally_row=0)
        return dict(pos=eng.pos[eng.parity], neg=eng.neg[eng.parity], tally=eng.tally.float(), histogram=eng.counts)
    if kind == "gradient":
        ks, grad, _ = pkg.ks_and_gradient(state["config"], checkpoint_every=case["checkpoint_every"],
                                          **_gradient_options(case))
        return dict(ks=np.float32(ks), gradient=grad.astype(np.float32))
    return _record(pkg.run_batched_b200(state["configs"]), case["dtype"], ks=True, fields=False)


def _wants_fields(case):
    # the study of two carrier species asks for k_s and the tallies: once its
    # faster carrier has left the gap, what float32 holds of it is underflow
    return "max_steps" not in case and not case["two_species"]


def _gradient_options(case):
    # a run cut short is launched with the library's own shapes: tuning a
    # large grid would take longer than these few steps
    return dict(max_steps=case["max_steps"], shape=dict(variant="auto")) if "max_steps" in case else {}


def _record(results, dtype, ks, fields):
    t = np.float64 if dtype == "float64" else np.float32
    join = lambda f: np.concatenate([np.ravel(f(r)) for r in results]).astype(t)  # noqa: E731
    out = dict(injected=join(lambda r: r.injected_positive), recombined=join(lambda r: r.recombination),
               n_positive=join(lambda r: r.n_positive), n_negative=join(lambda r: r.n_negative),
               f_t=join(lambda r: r.f_t),
               histogram=np.concatenate([np.ravel(r.track_density_xy) for r in results]).astype(np.int64))
    if ks:
        out["ks"] = join(lambda r: np.array([r.ks]))
    if fields:
        out["positive"], out["negative"] = (a.astype(t) for a in (results[0].positive_array, results[0].negative_array))
    return out


# --- what a pass cannot do without -------------------------------------------


def _steps_of(case, s):
    if case["kind"] == "segment":
        return case["pulse_steps"] + case["idle_steps"]
    return min(s["steps"], case.get("max_steps") or s["steps"])


def _step_work(s, steps, dtype):
    """27 operations a voxel and step (two seven-point stencils, the sink, the
    tallies). Fields beyond the L2 are read and written every step; smaller
    ones are read and written once."""
    es = 8 if dtype == "float64" else 4
    vox = (s["n"] - 2) ** 2 * (s["nzb"] - 2)
    passes = steps if 2 * es * vox > L2_BYTES else 1
    return dict(bytes=4.0 * es * vox * passes, flops=27.0 * vox * steps)


def work(case):
    if case["kind"] == "batch":
        ws = []
        for kw in _sweep_kwargs(case, 1):
            s = _scalars(kw)
            ws.append(_step_work(s, s["steps"], case["dtype"]))
        return dict(bytes=sum(w["bytes"] for w in ws), flops=sum(w["flops"] for w in ws))
    s = _scalars(_kwargs(case, 1))
    w = _step_work(s, _steps_of(case, s), case["dtype"])
    if case["kind"] == "gradient":
        # the forward solve, and per reverse step the state and lambda read and lambda written (24 bytes, 60 operations)
        return dict(bytes=w["bytes"] * 2.5, flops=w["flops"] * (1.0 + 60.0 / 27.0))
    return w


# --- the same results in plain 64-bit torch and numpy -------------------------


def _scalars(kw):
    """The numbers of a run that its inputs imply."""
    h = kw["grid_size_um"] * 1e-4
    e_field = kw["voltage_V"] / kw["electrode_gap_cm"]
    mu = (kw.get("mu_positive_cm2_Vs", 1.65), kw.get("mu_negative_cm2_Vs", 1.65))
    diff = (kw.get("D_positive_cm2_s", 3.7e-2), kw.get("D_negative_cm2_s", 3.7e-2))
    n = int(round(2 * kw["sampled_radius_cm"] / h)) + 8
    no_z = int(round(kw["electrode_gap_cm"] / h))
    dt = 1.0
    while True:
        dt /= 1.01
        if all(6 * (d * dt / h**2) + (m * e_field * dt / h) ** 2 <= 1 for d, m in zip(diff, mu)):
            break
    separation = int(kw["electrode_gap_cm"] / (2.0 * min(mu) * e_field * dt))
    bins = np.arange(0.0, kw["pulse_duration_s"] + dt, dt)
    pulse_steps = len(bins) - 1
    period = int(round(1.0 / kw["repetition_rate_hz"] / dt))
    n_eV = LET_KEV_UM * 1e7 / 34.2
    inst = kw["dose_rate_Gy_s"] / kw["repetition_rate_hz"] / kw["pulse_duration_s"]
    fluence_rate = inst * 6.241e15 * (1.225 * 1e-6) / (LET_KEV_UM * 1e4)
    area = math.pi * kw["sampled_radius_cm"] ** 2
    return dict(h=h, n=n, no_z=no_z, nze=3, nzb=no_z + 6, dt=dt, e_field=e_field, mu=mu, diff=diff, gap=kw["electrode_gap_cm"],
                volts=kw["voltage_V"], bins=bins, pulse_steps=pulse_steps, period=period, pulses=kw["n_pulses"],
                steps=(kw["n_pulses"] - 1) * period + pulse_steps + int(round(2.0 * separation)),
                pulse_s=kw["pulse_duration_s"], mid=n / 2.0, inner=n / 2.0 - 4, G=n_eV / (math.pi * TRACK_RADIUS_CM**2),
                h2b2=h**2 / TRACK_RADIUS_CM**2, cut=10.0 * (TRACK_RADIUS_CM / math.sqrt(2.0)) / h,
                tracks=max(1, int(round(fluence_rate * kw["pulse_duration_s"] * area))),
                reflecting=kw["lateral_boundary"] == "reflecting", seed=kw["seed"])


def _disc(rng, s, count):
    xs, ys = np.empty(0), np.empty(0)
    while len(xs) < count:
        u = rng.random((count + 64, 2)) * s["n"]
        u = u[((u - s["mid"]) ** 2).sum(1) <= s["inner"] ** 2]
        xs, ys = np.concatenate([xs, u[:, 0]]), np.concatenate([ys, u[:, 1]])
    return xs[:count], ys[:count]


def _segment_tracks(case, s, seed):
    rng = np.random.default_rng([int(seed), 77])
    counts = np.zeros(_steps_of(case, s), dtype=np.int64)
    counts[: case["pulse_steps"]] = rng.poisson(s["tracks"] / s["pulse_steps"], case["pulse_steps"])
    offsets = np.concatenate([[0], np.cumsum(counts)])
    return (offsets, *_disc(rng, s, int(offsets[-1])))


def _fill(field, s, seed):
    """Densities of a pulse under way, in the gap; the wall columns mirror their neighbours."""
    g = torch.Generator(device=field.device).manual_seed(seed)
    gap = torch.empty((s["n"], s["n"], s["no_z"]), dtype=field.dtype, device=field.device)
    field.zero_()
    field[:, :, s["nze"] : s["nze"] + s["no_z"]] = gap.uniform_(0.6e9, 1.4e9, generator=g)
    for a, b in ((0, 1), (-1, -2)):
        field[a] = field[b]
    for a, b in ((0, 1), (-1, -2)):
        field[:, a] = field[:, b]


def _plain_tracks(s):
    """A run's tracks per step and centres, drawn as the schedule defines them."""
    rng = np.random.default_rng(s["seed"])
    t = np.cumsum(rng.random(s["tracks"]))
    t = t / t[-1] * s["pulse_s"]
    one = np.histogram(t, s["bins"])[0]
    counts = np.zeros(s["steps"], dtype=np.int64)
    for p in range(s["pulses"]):
        counts[p * s["period"] : p * s["period"] + len(one)] += one
    total = int(counts.sum())
    xs, ys = [], []
    have = 0
    while have < total:
        u = rng.random((max(4096, 2 * (total - have)), 2)) * s["n"]
        u = u[(u[:, 0] - s["mid"]) ** 2 + (u[:, 1] - s["mid"]) ** 2 <= s["inner"] ** 2]
        xs.append(u[:, 0])
        ys.append(u[:, 1])
        have += len(u)
    return np.concatenate([[0], np.cumsum(counts)]), np.concatenate(xs)[:total], np.concatenate(ys)[:total]


def _plain_density(s, x, y):
    """G times the step's truncated Gaussians, [n, n]."""
    grid = torch.arange(s["n"], dtype=torch.float64, device=x.device)

    def factor(c):
        d = grid[None, :] - c[:, None]
        inside = (grid >= torch.ceil(c - s["cut"])[:, None]) & (grid <= torch.floor(c + s["cut"])[:, None])
        return torch.where(inside, torch.exp(-d * d * s["h2b2"]), 0.0)

    return s["G"] * (factor(x).T @ factor(y))


def _weights(s, mu, diff, volts, alpha):
    w = []
    for m, d in zip(mu, diff):
        c, q = m * (volts / s["gap"]) * s["dt"] / s["h"], d * s["dt"] / s["h"] ** 2
        w.append((q, q + c * (c + 1.0) / 2.0, q + c * (c - 1.0) / 2.0, 1.0 - c * c - 6.0 * q))
    return w[0], w[1], alpha * s["dt"]


def _plain_step(s, w, scored, P, N, dens):
    """(P, N, injected, recombined, n+, n-) after one step."""
    injected = 0.0
    if dens is not None:
        layer = torch.zeros(s["nzb"], dtype=torch.float64, device=P.device)
        layer[s["nze"] : s["nze"] + s["no_z"]] = 1.0
        add = dens[:, :, None] * layer
        P, N = P + add, N + add
        injected = (dens[1:-1, 1:-1] * scored).sum() * s["no_z"]
    (pl, pm, pp, pc), (nl, nm, np_, nc), a = w
    I = (slice(1, -1), slice(1, -1))
    rec = a * P[I + (slice(1, -1),)] * N[I + (slice(1, -1),)]
    out = []
    for U, lat, below, above, cen in ((P, pl, pm, pp, pc), (N, nl, np_, nm, nc)):
        k = slice(1, -1)
        side = U[2:, 1:-1, k] + U[:-2, 1:-1, k] + U[1:-1, 2:, k] + U[1:-1, :-2, k]
        V = below * U[1:-1, 1:-1, :-2] + above * U[1:-1, 1:-1, 2:] + lat * side + cen * U[I + (k,)] - rec
        V = torch.nn.functional.pad(V, (1, 1))
        if s["reflecting"]:
            V = torch.cat([V[:1], V, V[-1:]], 0)
            V = torch.cat([V[:, :1], V, V[:, -1:]], 1)
        else:
            V = torch.cat([U[:1, 1:-1], V, U[-1:, 1:-1]], 0)
            V = torch.cat([U[:, :1], V, U[:, -1:]], 1)
        out.append(V)
    gap = slice(s["nze"], s["nze"] + s["no_z"])
    sums = [(t * scored[:, :, None]).sum() for t in (rec[:, :, s["nze"] - 1 : s["nze"] - 1 + s["no_z"]],
                                                     out[0][I + (gap,)], out[1][I + (gap,)])]
    return (*out, injected, *sums)


def _plain_scored(s, dev):
    i = torch.arange(1, s["n"] - 1, dtype=torch.float64, device=dev) - s["mid"]
    return ((i[:, None] ** 2 + i[None, :] ** 2) < s["inner"] ** 2).double()


def _plain_run(s, offsets, xs, ys, P, N, w):
    dev = P.device
    scored = _plain_scored(s, dev)
    x, y = torch.from_numpy(xs).to(dev), torch.from_numpy(ys).to(dev)
    rows = []
    with torch.no_grad():
        for k in range(len(offsets) - 1):
            o0, o1 = int(offsets[k]), int(offsets[k + 1])
            dens = _plain_density(s, x[o0:o1], y[o0:o1]) if o1 > o0 else None
            P, N, *sums = _plain_step(s, w, scored, P, N, dens)
            rows.append(torch.stack([torch.as_tensor(t, dtype=torch.float64, device=dev) for t in sums]))
    return P, N, torch.stack(rows)


def _plain_histogram(s, xs, ys):
    return np.bincount(xs.astype(np.int64) * s["n"] + ys.astype(np.int64), minlength=s["n"] ** 2)


def _plain_gradient(s, case, offsets, xs, ys, dev):
    from torch.utils.checkpoint import checkpoint

    scored = _plain_scored(s, dev)
    x, y = torch.from_numpy(xs).to(dev), torch.from_numpy(ys).to(dev)
    theta = torch.tensor([ALPHA, *s["mu"], *s["diff"], s["volts"]], dtype=torch.float64, device=dev, requires_grad=True)
    P = torch.zeros((s["n"], s["n"], s["nzb"]), dtype=torch.float64, device=dev)
    N = torch.zeros_like(P)
    total = len(offsets) - 1
    length = max(1, min(24, int(20e9 / (30 * P.numel() * 8))))

    def stretch(P, N, theta, k0, k1):
        w = _weights(s, (theta[1], theta[2]), (theta[3], theta[4]), theta[5], theta[0])
        injected = torch.zeros((), dtype=torch.float64, device=dev)
        recombined = torch.zeros((), dtype=torch.float64, device=dev)
        for k in range(k0, k1):
            o0, o1 = int(offsets[k]), int(offsets[k + 1])
            dens = _plain_density(s, x[o0:o1], y[o0:o1]) if o1 > o0 else None
            P, N, i, r, _, _ = _plain_step(s, w, scored, P, N, dens)
            injected, recombined = injected + i, recombined + r
        return P, N, injected, recombined

    I = R = 0.0
    for k0 in range(0, total, length):
        P, N, i, r = checkpoint(stretch, P, N, theta, k0, min(k0 + length, total), use_reentrant=False)
        I, R = I + i, R + r
    ks = I / (I - R)
    ks.backward()
    return dict(ks=ks.detach().cpu().numpy(), gradient=theta.grad.cpu().numpy())


def exact(case, seed):
    dev = torch.device("cuda")
    kws = _sweep_kwargs(case, seed) if case["kind"] == "batch" else [_kwargs(case, seed)]
    ss = [_scalars(kw) for kw in kws]
    cost = sum(_steps_of(case, s) * (7e-4 + s["n"] ** 2 * s["nzb"] * 4e-10) for s in ss)
    if cost * (4 if case["kind"] == "gradient" else 1) > 18.0:
        return None
    if case["kind"] == "segment":
        s = ss[0]
        offsets, xs, ys = _segment_tracks(case, s, seed)
        kp = (s["nzb"] + 7) // 8 * 8
        P, N = (torch.zeros((s["n"], s["n"], s["nzb"]), dtype=torch.float32, device=dev) for _ in range(2))
        _fill(P, s, 2 * int(seed))
        _fill(N, s, 2 * int(seed) + 1)
        w = _weights(s, s["mu"], s["diff"], s["volts"], ALPHA)
        P, N, rows = _plain_run(s, offsets, xs, ys, P.double(), N.double(), w)
        pad = lambda f: torch.nn.functional.pad(f, (0, kp - s["nzb"]))  # noqa: E731
        return dict(pos=pad(P), neg=pad(N), tally=rows, histogram=None)
    parts = []
    for s in ss:
        offsets, xs, ys = _plain_tracks(s)
        steps = _steps_of(case, s)
        offsets = offsets[: steps + 1]
        xs, ys = xs[: offsets[-1]], ys[: offsets[-1]]
        if case["kind"] == "gradient":
            return _plain_gradient(s, case, offsets, xs, ys, dev)
        P = torch.zeros((s["n"], s["n"], s["nzb"]), dtype=torch.float64, device=dev)
        w = _weights(s, s["mu"], s["diff"], s["volts"], ALPHA)
        P, N, rows = _plain_run(s, offsets, xs, ys, P, torch.zeros_like(P), w)
        rows = np.concatenate([rows.cpu().numpy(), np.zeros((s["steps"] - steps, 4))])
        I, R = np.cumsum(rows[:steps, 0]), np.cumsum(rows[:steps, 1])
        f_t = np.ones(s["steps"])
        np.divide(I - R, I, out=f_t[:steps], where=I != 0)
        parts.append(dict(injected=rows[:, 0], recombined=rows[:, 1], n_positive=rows[:, 2], n_negative=rows[:, 3],
                          f_t=f_t, ks=np.array([1.0 / f_t[-1]])))
    out = {k: np.concatenate([p[k] for p in parts]) for k in parts[0]}
    out["histogram"] = None
    if "max_steps" in case:
        del out["ks"]
    elif case["kind"] == "run" and _wants_fields(case):
        out["positive"], out["negative"] = P.cpu().numpy(), N.cpu().numpy()
    return out
