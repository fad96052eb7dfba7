"""The work that users of this package have it do, as cases that can be timed.

A case is a dict of plain values.  ``listed()`` gives the fixed ones, ``draw(rng)``
one more of the same ranges, ``prepare(case, seed)`` what a program holds before the
call, ``run(state)`` one pass through the public entry points, ``work(case)`` the
bytes and operations that the pass cannot do without, and ``exact(case, seed)`` the
same outputs in 64 bits from plain torch.

Kinds of case:
  pass   solver.propagate: one crystal pass (Heun or RK23 schedule)
  mex    solver.opo_mex_batch: the drop-in solver call, its Ap and step records
         included; several pulses share one schedule
  sweep  solver.propagate (or a recorded graph of it) over pulses of uneven grids
         and crystals
  opo    opo.OpticalSim.run: round trips of a synchronously pumped cavity
  wide   solver.propagate_fp64 and solver.propagate_f32x2
  fibre  gnlse.propagate: a batch of fibre propagations
  trip   a network trip of the fast-forward loop: encode, FNO.forward, step
  train  FNO.backward: loss and gradients of a minibatch

Crystals are short (20 to 200 um) so that a pass takes milliseconds; the per-step work
is that of the long crystals.  Grids keep the sample spacing of 6 ps / 2^13.
"""
import dataclasses
import math

import numpy as np
import torch

from optifax_gb300 import _native as nat
from optifax_gb300 import fastforward as ff
from optifax_gb300 import gnlse, opo, surrogate, sweep
from optifax_gb300 import physics as ph
from optifax_gb300 import solver as sv

DEV = "cuda:0"
DT = 6e-12 / 2 ** 13
TRIP_POINTS = 2 ** 14


def listed():
    return [
        # the smallest grid and a short crystal: a call of about a millisecond
        {"name": "pass_512", "kind": "pass", "n": 512, "um": 30.0, "watts": 1.0, "fs": 100.0, "method": "heun"},
        # the drop-in solver call as the host program makes it, one pulse
        {"name": "mex_4096", "kind": "mex", "n": 4096, "um": 101.3, "watts": 2.0, "fs": 200.0, "pulses": 1},
        # the same with a batch of pulses on one shared schedule
        {"name": "mex_2048x6", "kind": "mex", "n": 2048, "um": 60.0, "watts": 1.5, "fs": 150.0, "pulses": 6},
        # the higher-order schedule at a tight tolerance (2^13 points over 6 ps)
        {"name": "rk23_8192", "kind": "pass", "n": 8192, "um": 60.0, "watts": 1.0, "fs": 200.0, "method": "rk23"},
        # the cavity of the default benchmark (2^14 points over 12 ps), a shorter crystal, three trips
        {"name": "opo_16384", "kind": "opo", "um": 100.0, "watts": 2.0, "fs": 200.0, "trips": 3, "cavities": 1},
        # the largest grid: a chirped grating, one pulse
        {"name": "pass_65536", "kind": "pass", "n": 65536, "um": 120.0, "watts": 3.0, "fs": 100.0, "method": "heun"},
        # a parameter sweep of uneven grids (2^12 to 2^16) and crystals that fills the GPU
        {"name": "sweep_48", "kind": "sweep", "pulses": 48, "um_lo": 20.0, "um_hi": 110.0, "graph": False},
        # the plain FP64 solver
        {"name": "fp64_4096", "kind": "wide", "n": 4096, "um": 50.0, "watts": 2.0, "fs": 200.0, "pulses": 1,
         "entry": "fp64"},
        # the float-float solver for high-gain passes
        {"name": "f32x2_16384", "kind": "wide", "n": 16384, "um": 50.0, "watts": 2.0, "fs": 200.0, "pulses": 1,
         "entry": "f32x2"},
        # a power scan of fibre pulses, one per SM
        {"name": "fibre_152x4096", "kind": "fibre", "n": 4096, "pulses": 152, "mm": 5.0, "saves": 5},
        # one network trip of the fast-forward loop: small kernels, latency and launches count (weights
        # of the initial distribution: a trained network magnifies the last bits of a BF16 rounding)
        {"name": "trip_1", "kind": "trip", "spectra": 1, "repr": "env"},
        # a training minibatch of the surrogate
        {"name": "train_32", "kind": "train", "batch": 32, "bins": 4096},
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["pass", "pass", "mex", "sweep", "opo", "wide", "fibre", "trip", "train"])
    watts, fs = round(rng.uniform(0.5, 3.0), 3), round(rng.uniform(100.0, 300.0), 2)
    if kind == "pass":
        n = 2 ** rng.randint(9, 16)
        if rng.random() < 0.25 and n <= 16384:
            return {"kind": "pass", "n": n, "um": round(_log(rng, 15, 60), 1), "watts": watts, "fs": fs, "method": "rk23"}
        return {"kind": "pass", "n": n, "um": round(_log(rng, 20, 120), 1), "watts": watts, "fs": fs, "method": "heun"}
    if kind == "mex":
        n = 2 ** rng.randint(9, 14)
        most = max(1, min(16, 96 * 4096 // n // 4))
        return {"kind": "mex", "n": n, "um": round(_log(rng, 20, 110), 1), "watts": watts, "fs": fs,
                "pulses": rng.randint(1, most) if rng.random() < 0.5 else 1}
    if kind == "sweep":
        return {"kind": "sweep", "pulses": max(3, int(_log(rng, 3, 48))), "um_lo": round(rng.uniform(15, 25), 1),
                "um_hi": round(rng.uniform(40, 110), 1), "graph": rng.random() < 0.5}
    if kind == "opo":
        return {"kind": "opo", "um": round(rng.uniform(30, 100), 1), "watts": watts, "fs": fs, "trips": rng.randint(1, 3),
                "cavities": rng.randint(1, 8)}
    if kind == "wide":
        entry = rng.choice(["fp64", "f32x2"])
        n = 2 ** rng.randint(9, 15 if entry == "f32x2" else 14)
        return {"kind": "wide", "n": n, "um": round(_log(rng, 15, 50), 1), "watts": watts, "fs": fs,
                "pulses": rng.choice([1, 1, 2]) if n <= 8192 else 1, "entry": entry}
    if kind == "fibre":
        return {"kind": "fibre", "n": 2 ** rng.randint(9, 12), "pulses": max(1, int(_log(rng, 1, 153))),
                "mm": round(_log(rng, 1, 5), 2), "saves": rng.randint(2, 9)}
    if kind == "trip":
        k = rng.choice([1, rng.randint(2, 32)])
        return {"kind": "trip", "spectra": k, "repr": "bins" if k == 1 else rng.choice(["env", "bins"])}
    return {"kind": "train", "batch": max(1, int(_log(rng, 1, 33))), "bins": 64 * rng.randint(8, 64)}


# ---- inputs -------------------------------------------------------------------------
def _gpu(x, dtype):
    return torch.from_numpy(np.ascontiguousarray(np.asarray(x).astype(dtype))).to(DEV)


def _jitter(case, seed):
    r = np.random.default_rng(seed)
    return case["watts"] * r.uniform(0.98, 1.02), case["fs"] * r.uniform(0.98, 1.02)


def _crystal_inputs(case, seed, pulses=1):
    """(SolverInputs, input fields (pulses, n) complex128) of a poled crystal behind its face."""
    n = case["n"]
    watts, fs = _jitter(case, seed)
    win = ph.SimWindow(1040e-9, n, n * DT)
    length = case["um"] * 1e-6
    period = ("chirpedgrating", 28e-6, 32e-6, 1.0, 0.1e-6) if n == 65536 and length > 50e-6 else 30e-6
    bounds = (1e-4 / 20, 1e-4) if case.get("method") == "rk23" else (2.5e-3, 5e-2)
    si = ph.solver_inputs(ph.Crystal(length, period), win, error_bounds=bounds)
    tau = min(fs * 1e-15, win.temporal_range / 12)      # keep the pulse clear of the absorber
    fields = []
    for b in range(pulses):
        pump = ph.sech_pump(win, 1040e-9, tau, watts * (1.0 + 0.1 * b))
        noise = ph.photon_noise(win, 1000 * seed + b, mask=ph.window_transmission(win))
        fields.append(np.fft.ifft(np.fft.fft(np.fft.fftshift(pump + noise)) * np.sqrt(1.0 / si.n_index)))
    return si, np.array(fields)


def _network_inputs(batch, bins, seed):
    """Network inputs and targets as encoded trips give them: a pump and a signal envelope each
    (signal at unit RMS), the signal's log-level and the bin coordinate."""
    g = torch.Generator(device=DEV).manual_seed(seed)
    rnd = lambda *s: torch.rand(*s, generator=g, device=DEV)  # noqa: E731
    t = torch.linspace(-1, 1, bins, device=DEV)

    def envelope():
        u = (t - 0.2 * (rnd(batch, 1) - 0.5)) / (0.03 + 0.05 * rnd(batch, 1))
        ph_ = 6.2832 * rnd(batch, 1) + 3 * (rnd(batch, 1) - 0.5) * u
        a = (0.5 + 0.5 * rnd(batch, 1)) / torch.cosh(u)
        noise = 0.01 * torch.randn(2, batch, bins, generator=g, device=DEV)
        return a * torch.cos(ph_) + noise[0], a * torch.sin(ph_) + noise[1]

    pr, pi = envelope()
    sr, si = envelope()
    rms = (sr ** 2 + si ** 2).mean(dim=1, keepdim=True).sqrt()
    lev = (-2 * rnd(batch, 1)).expand(batch, bins)
    x = torch.stack([pr, pi, sr / rms, si / rms, lev, torch.arange(bins, device=DEV).expand(batch, bins) / bins], dim=1)
    qr, qi = envelope()
    t_ = torch.stack([0.8 * pr, 0.8 * pi, (sr + 0.4 * qr) / rms, (si + 0.4 * qi) / rms], dim=1)
    w = 1.0 / t_.pow(2).mean(dim=(1, 2))
    return x.float().contiguous(), t_.float().contiguous(), w.float().contiguous()


def _trip_inputs(case, seed):
    """Crystal-input spectra of a running cavity: the pump and a signal pulse in the fed-back band."""
    spec = opo.CavitySpec()
    a = opo.build_cavity(spec)
    crop = ff.make_env_crop(a.win, a.pump, signal_band_nm=spec.signal_band_nm) if case["repr"] == "env" else \
        ff.make_crop(a.win, float(np.max(np.abs(a.pump))))
    r = np.random.default_rng(seed)
    f = np.fft.ifftshift(a.win.rel_freqs) + a.win.f0
    Y = []
    for _ in range(case["spectra"]):
        fs_, bw = r.uniform(185e12, 205e12), r.uniform(2e12, 6e12)
        s = np.exp(-((f - fs_) / bw) ** 2 + 1j * (2 * np.pi * r.uniform() + r.normal() * ((f - fs_) / bw) ** 2))
        Y.append(a.pump * r.uniform(0.8, 1.2) + r.uniform(0.1, 0.5) * np.max(np.abs(a.pump)) * s)
    si = a.si
    D = np.asarray(si.alpha, np.float64) ** si.n_steps * np.exp(-1j * np.asarray(si.beta, np.float64) * si.n_steps)
    return crop, np.array(Y), a.feedback, a.pump, D


def _cavities(case, seed):
    watts, fs = _jitter(case, seed)
    return [opo.CavitySpec(n_points=2 ** 14, window=12e-12, crystal_length=case["um"] * 1e-6, pump_power=watts * (1 + 0.05 * i),
                           pump_tau=fs * 1e-15, seed=1000 * seed + i) for i in range(case["cavities"])]


def _sweep_specs(case, seed):
    lo, hi = case["um_lo"] * 1e-6, case["um_hi"] * 1e-6
    grids = sweep.uneven_sweep_instances(case["pulses"], seed=2)          # the sizes belong to the case
    insts = sweep.uneven_sweep_instances(case["pulses"], seed=seed, length_range=(lo, hi))
    return sweep.build_specs_device([dataclasses.replace(i, n_points=g.n_points) for i, g in zip(insts, grids)])


def _fibre(case, seed):
    n = case["n"]
    T = np.arange(-n // 2, n // 2) * (6e-12 / 4096)
    w0 = 2 * np.pi * 299792458.0 / 835e-9
    ops = gnlse.fibre_operators(T, w0, 0.11, [-1.183e-26, 8.1e-41, -9.5e-56], 0.0, 0.18, gnlse.raman_response(T))
    r = np.random.default_rng(seed)
    p0 = np.sort(r.uniform(1e3, 1e4, case["pulses"]))
    A = np.sqrt(p0)[:, None] / np.cosh(T / 28.4e-15)
    return ops, _gpu(A, np.complex64), w0


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case}
    if kind == "pass":
        si, E = _crystal_inputs(case, seed)
        s["spec"] = sv.PulseSpec(E=_gpu(E[0], np.complex64), alpha=_gpu(si.alpha, np.float32), beta=_gpu(si.beta, np.float32),
                                 G=_gpu(si.G, np.float32), w0=si.w0, bdiffw0=si.bdiffw0, h=si.h, dt=si.dt,
                                 max_err=si.max_err, min_err=si.min_err, sel=si.sel, n_steps=si.n_steps)
    elif kind == "mex":
        si, E = _crystal_inputs(case, seed, case["pulses"])
        G = si.G if case["pulses"] == 1 else np.stack([si.G] * case["pulses"])
        chunks = sv.n_chunks(si.n_steps, si.sel)
        s.update(si=si, E=_gpu(E, np.complex64), alpha=_gpu(si.alpha, np.float32), beta=_gpu(si.beta, np.float32),
                 G=_gpu(G, np.float32), Ap=torch.zeros((len(E), chunks, case["n"]), dtype=torch.complex64, device=DEV),
                 steps=torch.zeros(si.n_steps, dtype=torch.float32, device=DEV))
    elif kind == "sweep":
        s["specs"] = _sweep_specs(case, seed)
        if case["graph"]:
            s["graph"] = sv.propagate_graph(s["specs"])
    elif kind == "opo":
        s["sims"] = [opo.OpticalSim(c) for c in _cavities(case, seed)]
        s["fields"] = [sim.field for sim in s["sims"]]
    elif kind == "wide":
        si, E = _crystal_inputs(case, seed, case["pulses"])
        s.update(si=si, E=_gpu(E, np.complex128), alpha=_gpu(si.alpha, np.float64), beta=_gpu(si.beta, np.float64),
                 G=_gpu(si.G, np.float64))
    elif kind == "fibre":
        s["ops"], s["A"], s["w0"] = _fibre(case, seed)
    elif kind == "trip":
        crop, Y, fb, pump, D = _trip_inputs(case, seed)
        s.update(crop=crop, Y=_gpu(Y, np.complex64), fb=_gpu(fb, np.complex64), pump=_gpu(pump, np.complex64),
                 D=_gpu(D, np.complex64), net=surrogate.FNO(crop.n_bins, max_batch=case["spectra"], params=surrogate.init_params(seed)))
    else:
        s["net"] = surrogate.FNO(case["bins"], max_batch=case["batch"], params=surrogate.init_params(seed))
        s["x"], s["t"], s["w"] = _network_inputs(case["batch"], case["bins"], seed)
        s["grads"] = torch.empty(surrogate.N_PARAMS, dtype=torch.float32, device=DEV)
    return s


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "pass":
        rk = case["method"] == "rk23"
        outs, _ = sv.propagate([state["spec"]], method=nat.RK23 if rk else nat.HEUN,
                               variant=nat.VARIANT_ODE23 if rk else nat.VARIANT_BATCH_XTAL, want_stats=False)
        return outs
    if kind == "mex":
        si = state["si"]
        return sv.opo_mex_batch(state["E"], state["alpha"], state["G"], si.w0, si.bdiffw0, si.h, si.n_steps, si.dt,
                                state["beta"], si.max_err, si.min_err, si.sel, state["Ap"], state["steps"])
    if kind == "sweep":
        if case["graph"]:
            state["graph"].launch()
            return state["graph"].outputs
        return sv.propagate(state["specs"], want_stats=False)[0]
    if kind == "opo":
        for sim, field in zip(state["sims"], state["fields"]):
            sim.field = field
        res = opo.run_many(state["sims"], case["trips"], host_out=False, history=True)
        return [[r.field, r.history] for r in res]
    if kind == "wide":
        si = state["si"]
        entry = sv.propagate_fp64 if case["entry"] == "fp64" else sv.propagate_f32x2
        A, _, _ = entry(state["E"], state["alpha"], state["beta"], state["G"], w0=si.w0, bdiffw0=si.bdiffw0, h=si.h,
                        dt=si.dt, n_steps=si.n_steps, max_err=si.max_err, min_err=si.min_err, sel=si.sel)
        return A
    if kind == "fibre":
        r = gnlse.propagate(state["ops"], state["A"], case["mm"] * 1e-3, case["saves"], w0=state["w0"])
        return [r.AT, r.AW]
    if kind == "trip":
        x, sigma = ff.encode(state["Y"], state["crop"])
        y = state["net"].forward(x)
        if case["spectra"] > 1:
            return [x, sigma, y]
        X = torch.empty(TRIP_POINTS, dtype=torch.complex64, device=DEV)
        Y = ff.step(state["crop"], state["fb"], state["pump"], None, y=y, sigma=sigma, lin=state["D"], X_out=X)
        return [x, sigma, y, X, Y]
    loss = state["net"].backward(state["x"], state["t"], grads=state["grads"], sample_w=state["w"])
    return [loss, state["grads"]]


# ---- what a pass cannot do without ---------------------------------------------------
def _pass_work(n, um, item=4):
    steps = um / 0.1
    attempts = steps / 2.2                     # measured over these crystals: two to three z-samples a step
    return item * (6 * n + steps), attempts * n * (10 * math.log2(n) + 60)


def work(case):
    kind = case["kind"]
    if kind in ("pass", "mex", "wide"):
        b, f = _pass_work(case["n"], case["um"], 8 if kind == "wide" else 4)
        k = case.get("pulses", 1)
        if kind == "mex":
            b += 8 * 5 * case["n"]
        if case.get("method") == "rk23":
            f *= 3.0
        return {"bytes": k * b, "flops": k * f}
    if kind == "sweep":
        got = [_pass_work(2 ** p, 0.5 * (case["um_lo"] + case["um_hi"])) for p in range(12, 17)]
        k = case["pulses"] / 5
        return {"bytes": k * sum(b for b, _ in got), "flops": k * sum(f for _, f in got)}
    if kind == "opo":
        b, f = _pass_work(TRIP_POINTS, case["um"])
        k = case["cavities"]
        return {"bytes": k * (b + 8 * TRIP_POINTS * (3 + case["trips"])), "flops": k * f * case["trips"]}
    if kind == "fibre":
        n, steps = case["n"], 13.0 * case["mm"]          # a 1 to 10 kW scan: 6 to 14 steps per mm
        flops = 6 * steps * (20 * n * math.log2(n) + 40 * n)
        return {"bytes": case["pulses"] * 8 * n * (1 + 2 * case["saves"]), "flops": case["pulses"] * flops}
    b, bins = (case["spectra"], 4096) if kind == "trip" else (case["batch"], case["bins"])
    w, modes, layers = surrogate.W, surrogate.MODES, surrogate.NLAYER
    fwd = b * layers * (2 * bins * w * w + 8 * w * bins * modes + 8 * w * w * modes) + 20 * b * bins * w
    if kind == "trip":
        return {"bytes": 4 * (10 * b * bins) + 8 * b * TRIP_POINTS + 4 * surrogate.N_PARAMS, "flops": fwd}
    return {"bytes": 4 * (10 * b * bins) + 8 * surrogate.N_PARAMS, "flops": 3 * fwd}


# ---- the same in 64 bits --------------------------------------------------------------
def _absorber(n):
    i = torch.arange(n, dtype=torch.float64, device=DEV)
    f = torch.tanh(48.0 * (i - n / 2).abs() / n) ** 2
    return torch.where((i > 6 * (n // 16)) & (i < 10 * (n // 16)), f, torch.ones_like(f))


def _exact_pass(E, alpha, beta, G, p, rk=False):
    """(output fields, chunk spectra, step record, last spectrum) of pulses E (B, n) on one schedule."""
    B, n = E.shape
    S, sel, h, w0 = int(p.n_steps), float(p.sel), float(p.h), float(p.w0)
    E = E.to(torch.complex128)
    alpha, beta, G = alpha.double(), beta.double(), np.atleast_2d(G.double().cpu().numpy())
    i = torch.arange(n, dtype=torch.float64, device=DEV)
    jt = i if rk else torch.where(i > n // 2, i - n // 2, i + n // 2)
    carrier = torch.polar(torch.ones_like(jt), torch.remainder(w0 * float(p.dt) * jt, 2 * math.pi))
    cs, absorb = 1.0 / (2.0 * float(p.dt) * w0), _absorber(n)

    def drive(A, z, k, s):
        e = carrier * complex(math.cos(-p.bdiffw0 * h * z), math.sin(-p.bdiffw0 * h * z))
        nl = A * A * e + 2.0 * (A.abs() ** 2) * e.conj()
        g = torch.from_numpy(s * h * G[:, k]).to(DEV)[:, None]
        return -1j * g * (nl - 1j * cs * (torch.roll(nl, -1, 1) - torch.roll(nl, 1, 1)))

    chunks = int(S / sel)
    if not rk and chunks * sel < S:
        chunks += 1
    limit = (n // 256) * 256 if rk else -(-n // 128) * 128
    Ap, record = torch.zeros((B, chunks, n), dtype=torch.complex128, device=DEV), torch.zeros(S, dtype=torch.float64)
    k, prev, s, cached, spec = 0.0, 4.0, 4.0, None, None
    K1 = drive(E, 0.0, 0, s) if rk else None
    for chunk in range(chunks):
        s, end = prev, (chunk + 1) * sel
        while k < end and (rk or k < S):
            ki = int(k)
            if rk:
                K2 = drive(E + 0.5 * K1, k + 0.5 * s, ki, s)
                K3 = drive(E + 0.75 * K2, k + 0.75 * s, ki, s)
                new = E + 4 / 9 * K3 + 1 / 3 * K2 + 2 / 9 * K1
                K4 = drive(new, k + s, ki, s)
                d = 2 * (K3 / 9 + K2 / 12 - 5 / 72 * K1 - K4 / 8)
            else:
                K1 = drive(E, k, ki, s)
                K2 = drive(E + K1, k + s, ki, s)
                new = E + 0.5 * (K1 + K2)
                d = 0.5 * (K2 - K1)
            a = new.abs()
            worst = float(torch.where(a > 0, 100.0 * d.abs() / (a + 1.0), torch.zeros_like(a)).max())
            big, grow = worst >= p.max_err, worst < p.min_err
            if big and s > 1 and k - s > 0:
                k, s = k - s, s - 1
                prev = s
                if rk:
                    K1 = drive(E, k + s, int(k), s)
            else:
                used = int(s)
                if ki < limit and ki < S:
                    record[ki] = used
                if k + s >= end and k < end - 1:
                    prev, s = s, end - k - 1
                else:
                    if grow and rk and k + 2 * s < end - 1:
                        s = 2 * s
                    elif grow and not rk and k + s + 1 < end - 1:
                        s += 1
                    prev = s
                if cached != used:
                    factor = torch.polar(alpha ** used, -torch.remainder(beta * used, 2 * math.pi))
                    cached = used
                spec = torch.fft.fft(new * absorb) * factor
                if not (k + s < end and (rk or k + s < S)):
                    Ap[:, chunk] = spec
                E = torch.fft.ifft(spec)
                if rk:
                    K1 = K4
            k += s
    return E, Ap, record.to(DEV), spec


def _exact_fibre(ops, A, length, saves, rtol=1e-5, atol=1e-12):
    """AT, AW of a batch: Dormand-Prince 5(4) with ode45's step rules, every pulse on its own schedule."""
    t64 = lambda v, dt: torch.from_numpy(np.ascontiguousarray(v)).to(DEV, dt)  # noqa: E731
    n, nb = ops.n, A.shape[0]
    L = 1j * t64(ops.B, torch.float64) - ops.alpha / 2
    Wt = t64(ops.W, torch.float64)
    RW = None if ops.RW is None else t64(ops.RW, torch.complex128)

    def rhs(z, y):
        ex = torch.exp(L * (z * length)[:, None])
        at = torch.fft.fft(y * ex)
        it = at.abs() ** 2
        g = it * (1 - ops.fr)
        if RW is not None:
            g = g + ops.dT * ops.fr * torch.fft.fft(torch.fft.ifft(it + 0j) * RW)
        return 1j * ops.gamma * Wt * torch.fft.ifft(at * g) / ex

    a = [[], [1 / 5], [3 / 40, 9 / 40], [44 / 45, -56 / 15, 32 / 9], [19372 / 6561, -25360 / 2187, 64448 / 6561, -212 / 729],
         [9017 / 3168, -355 / 33, 46732 / 5247, 49 / 176, -5103 / 18656], [35 / 384, 0, 500 / 1113, 125 / 192, -2187 / 6784, 11 / 84]]
    c = [0, 1 / 5, 3 / 10, 4 / 5, 8 / 9, 1, 1]
    e = [71 / 57600, 0, -71 / 16695, 71 / 1920, -17253 / 339200, 22 / 525, -1 / 40]

    def stages(z, y, k1, h, last):
        ks = [k1]
        for s in range(1, last + 1):
            ys = y + (h * length)[:, None] * sum(w * q for w, q in zip(a[s], ks) if w)
            ks.append(rhs(z + c[s] * h, ys))
        return ks

    norm = lambda v: torch.linalg.vector_norm(v, dim=1)  # noqa: E731
    y = torch.fft.ifft(A.to(torch.complex128))
    z, at = torch.zeros(nb, dtype=torch.float64, device=DEV), torch.zeros((2, nb, saves, n), dtype=torch.complex128, device=DEV)
    points = [i / (saves - 1) for i in range(saves)]

    def keep(rows, j, z_, y_):
        aw = y_ * torch.exp(L * (z_ * length)[:, None])
        at[0, rows, j] = torch.fft.fft(aw)
        at[1, rows, j] = torch.fft.fftshift(aw, dim=1) * ops.dT * n

    keep(torch.arange(nb, device=DEV), 0, z, y)
    k1 = rhs(z, y)
    thr = atol / rtol
    h = torch.clamp(0.8 * rtol ** 0.2 * norm(y).clamp_min(thr) / norm(k1).clamp_min(1e-300) / length, max=0.1)
    clean, fresh = torch.ones(nb, dtype=torch.bool, device=DEV), torch.ones(nb, dtype=torch.bool, device=DEV)
    hc = h.clone()
    rows = torch.arange(nb, device=DEV)
    while rows.numel():
        f = fresh[rows]
        hr = torch.where(f, h[rows].clamp(max=0.1), hc[rows])
        hr = torch.where(f & (1.1 * hr >= 1 - z[rows]), 1 - z[rows], hr)
        clean[rows] |= f
        zr, yr, kr = z[rows], y[rows], k1[rows]
        ks = stages(zr, yr, kr, hr, 6)
        yn = yr + (hr * length)[:, None] * sum(w * q for w, q in zip(a[6], ks) if w)
        ev = (hr * length)[:, None] * sum(w * q for w, q in zip(e, ks) if w)
        err = norm(ev) / torch.maximum(norm(yr), norm(yn)).clamp_min(thr)
        ok = err <= rtol
        end = torch.where(1 - (zr + hr) < 1e-12, torch.ones_like(zr), zr + hr)
        for j, pt in enumerate(points[1:], 1):
            hit = ok & (zr < pt - 1e-12) & (pt < end - 1e-12)
            if bool(hit.any()):
                r_, hs = rows[hit], pt - zr[hit]
                q = stages(zr[hit], yr[hit], kr[hit], hs, 5)
                keep(r_, j, zr[hit] + hs, yr[hit] + (hs * length)[:, None] * sum(w * v for w, v in zip(a[6], q) if w))
            on = ok & ((end - pt).abs() <= 1e-12)
            if bool(on.any()):
                keep(rows[on], j, end[on], yn[on])
        grow = 1.25 * (err / rtol) ** 0.2
        after = torch.where(clean[rows], torch.where(grow > 0.2, hr / grow, 5 * hr), hr)
        fail = torch.where(clean[rows], hr * (0.8 * (rtol / err) ** 0.2).clamp_min(0.1), hr / 2)
        h[rows], hc[rows] = torch.where(ok, after, h[rows]), torch.where(ok, hr, fail)
        clean[rows], fresh[rows] = clean[rows] & ok, ok
        g = rows[ok]
        z[g], y[g], k1[g] = end[ok], yn[ok], ks[6][ok]
        rows = rows[z[rows] < 1]
    return [at[0], at[1]]


def _exact_network(params, x, grad=False):
    """(y, parameters as one differentiable vector) of the network in 64 bits."""
    p = torch.as_tensor(np.asarray(params, dtype=np.float64), device=DEV).requires_grad_(grad)
    W, M, n = surrogate.W, surrogate.MODES, x.shape[-1]
    x = x.double()
    h = torch.einsum("ci,bix->bcx", p[:W * 6].view(W, 6), x) + p[surrogate.OFF_PB:surrogate.OFF_L0][None, :, None]
    for layer in range(surrogate.NLAYER):
        o = surrogate.OFF_L0 + layer * surrogate.LAYER_SIZE
        ws = torch.view_as_complex(p[o:o + surrogate.LAYER_WS].view(W, W, M, 2))
        wp = p[o + surrogate.LAYER_WS:o + surrogate.LAYER_WS + W * W].view(W, W)
        bias = p[o + surrogate.LAYER_WS + W * W:o + surrogate.LAYER_SIZE]
        T = torch.einsum("bcm,com->bom", torch.fft.rfft(h)[..., :M], ws)
        h = torch.fft.irfft(T, n=n) + torch.einsum("oc,bcx->box", wp, h) + bias[None, :, None]
        if layer < surrogate.NLAYER - 1:
            h = torch.nn.functional.gelu(h)
    q, qb = p[surrogate.OFF_Q:surrogate.OFF_QB].view(4, W), p[surrogate.OFF_QB:]
    return x[:, :4] + torch.einsum("jc,bcx->bjx", q, h) + qb[None, :, None], p


def _exact_trip(case, seed):
    crop, Y, fb, pump, D = _trip_inputs(case, seed)
    Y = _gpu(Y, np.complex64).to(torch.complex128)
    fb, pump, D = (_gpu(_gpu(v, np.complex64).cpu().numpy(), np.complex128) for v in (fb, pump, D))
    n, nb = crop.n_points, crop.n_bins
    bands = []
    if case["repr"] == "env":
        for kc, lo, hi in (crop.band[:3], crop.band[3:]):
            o = torch.arange(lo, hi, device=DEV)
            b = torch.zeros((Y.shape[0], nb), dtype=torch.complex128, device=DEV)
            b[:, o % nb] = Y[:, (kc + o) % n]
            bands.append(nb * torch.fft.ifft(b))
        sigma = (bands[1].abs() ** 2).mean(dim=1).sqrt()
    else:
        j = torch.arange(nb, device=DEV)
        crop_ = Y[:, (crop.k0 + j) % n]
        low = (j < crop.split).double()
        sigma = ((crop_.abs() ** 2) * low).sum(dim=1).div(crop.split).sqrt()
        bands = [crop_ * (1 - low), crop_ * low]
    p, s = bands[0] / crop.pump_scale, bands[1] / sigma[:, None]
    x = torch.stack([p.real, p.imag, s.real, s.imag, torch.log10(sigma / crop.pump_scale)[:, None].expand(-1, nb),
                     (torch.arange(nb, device=DEV, dtype=torch.float64) / nb).expand(len(Y), -1)], dim=1)
    y, _ = _exact_network(surrogate.init_params(seed), x)
    if case["spectra"] > 1:
        return [x, sigma, y]
    X = torch.zeros(n, dtype=torch.complex128, device=DEV)
    out = [torch.complex(y[0, 0], y[0, 1]) * crop.pump_scale, torch.complex(y[0, 2], y[0, 3]) * sigma[0]]
    if case["repr"] == "env":
        for v, (kc, lo, hi) in zip(out, (crop.band[:3], crop.band[3:])):
            o = torch.arange(lo, hi, device=DEV)
            X[(kc + o) % n] = (torch.fft.fft(v) / nb)[o % nb]
    else:
        j = torch.arange(nb, device=DEV)
        X[(crop.k0 + j) % n] = torch.where(j < crop.split, out[1], out[0])
    X = X * D
    return [x, sigma, y, X, X * fb + pump]


def exact(case, seed):
    kind = case["kind"]
    if kind in ("pass", "sweep"):
        s = prepare(dict(case, graph=False), seed)
        specs = [s["spec"]] if kind == "pass" else s["specs"]
        return [_exact_pass(p.E[None], p.alpha, p.beta, p.G, p, rk=case.get("method") == "rk23")[0][0] for p in specs]
    if kind in ("mex", "wide"):
        s = prepare(case, seed)
        A, Ap, record, _ = _exact_pass(s["E"], s["alpha"], s["beta"], s["G"], s["si"])
        return [A, Ap, record] if kind == "mex" else A
    if kind == "opo":
        got = []
        for sim in prepare(case, seed)["sims"]:
            field, history = sim.field[None].to(torch.complex128), []
            for _ in range(case["trips"]):
                spec = _exact_pass(field, sim.alpha, sim.beta, sim.G, sim.arrays.si)[3]
                history.append(spec[0])
                field = torch.fft.ifft(spec * sim.feedback + sim.pump)
            got.append([field[0], torch.stack(history)])
        return got
    if kind == "fibre":
        ops, A, _ = _fibre(case, seed)
        return _exact_fibre(ops, A, case["mm"] * 1e-3, case["saves"])
    if kind == "trip":
        return _exact_trip(case, seed)
    x, t, w = _network_inputs(case["batch"], case["bins"], seed)
    y, p = _exact_network(surrogate.init_params(seed), x, grad=True)
    loss = (w.double()[:, None, None] * (y - t.double()) ** 2).sum() / y.numel()
    loss.backward()
    return [loss.detach().reshape(1), p.grad]
