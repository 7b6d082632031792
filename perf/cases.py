"""The work that users of this framework have it do, as cases to be timed.

Each case is one call (or one step) through the package's public entry points,
over the range of sizes the repository's own workloads, tests and benchmark
use. listed() names fixed cases, draw() gives others of the same ranges,
prepare() makes what a user's program holds before the call, run() makes the
call, work() counts what it cannot do without, and exact() gives the call's
result in 64-bit torch, from the mathematics and without the package's kernels.

The kinds:

  point    Medium.vertical_displacement_multi: one frequency, a few ranges, the
           reference's formulation on its own default wavenumber grid. What an
           interactive query or a hierarchy check asks for; the smallest call.
  default  build_bank on the default grids (each bin its own): what the
           reference's bank builder runs.
  bank     Medium.bank_spectra on one shared wavenumber grid, host in and out:
           a bank of one soil at a fixed integration.
  plan     Plan.execute on a shared grid, the result left on the device: a
           program that builds bank after bank of one soil.
  batch    Batch.execute over uneven soils sharing ranges and grid, captured as
           one graph: banks for a soil survey.
  sobol    sobol.solve_metrics: the f-k solve at one sensor range and the
           trace metrics for rows of a Sobol design.
  impulse  DeviceBank.impulse_responses: footstep contacts served from a bank
           that stays on the device.
  disp     disp.modes_many: dispersion curves of a layered soil.
  predict  surrogate.Net.predict: a trained network answering soils at a sensor.
  train    surrogate.Net.train: optimiser steps on a filled data set.
  fdtd     fdtd.run: the finite-difference validator's shot.
"""
import importlib
import math

import numpy as np
import torch

gfk = importlib.import_module("co-simulation-of-seismic-sensors-and-ros-for-robotic-human-detection_b200")

FS = 1000.0  # sample rate of the synthetic workloads (Hz)
KMAX_SOILS = 2.5 * 2 * math.pi * 500.0 / 80.0  # wavenumber cut of the uneven-soil and Sobol workloads


def listed():
    return [
        # one response of the two-layer soil the reference times, four ranges, its default grid
        {"name": "point_2layer_4r", "kind": "point", "layers": 2, "nr": 4, "rmax": 20.0, "freq": 60.0},
        # the reference's own bank build: loam half-space, 614 bins to 300 Hz, 270 ranges to 40 m
        {"name": "default_loam_614x270", "kind": "default", "layers": 1, "nf": 614, "nr": 270, "rmax": 40.0,
         "fs": 2000.0, "samples": 4096},
        # the single-soil bank: 512 bins x 64 ranges, 4096 wavenumbers, FP64 sum, host to host
        {"name": "bank_512x64_fp64", "kind": "bank", "layers": 3, "nf": 512, "nr": 64, "nk": 4096, "split": False},
        # a bank of odd sizes with the split-precision sum
        {"name": "bank_301x93_split", "kind": "bank", "layers": 7, "nf": 301, "nr": 93, "nk": 3001, "split": True},
        # the graded-soil bank, the benchmark's workload: 2048 bins x 1024 ranges, 16384 wavenumbers
        {"name": "plan_2048x1024_split", "kind": "plan", "layers": 11, "nf": 2048, "nr": 1024, "nk": 16384,
         "split": True},
        # uneven soils of 2-12 layers, 256-2048 bins each, 128 ranges, one graph per execute
        {"name": "batch_64_soils_split", "kind": "batch", "soils": 64, "nr": 128, "nk": 8192, "split": True},
        # rows of a Sobol design: 512 bins at one range, metrics of the recorded trace
        {"name": "sobol_256_soils", "kind": "sobol", "soils": 256},
        # footstep contacts answered from a 1024-range bank
        {"name": "impulse_8192x1024", "kind": "impulse", "count": 1024, "samples": 4096, "nq": 8192, "length": 1024},
        # every mode of a ten-layer soil at 512 frequencies
        {"name": "disp_512f", "kind": "disp", "layers": 11, "nf": 512, "fmax": 200.0},
        # the network at one range and the trace's 512 bins
        {"name": "predict_2048_soils", "kind": "predict", "soils": 2048, "nr": 1},
        # optimiser steps at the training workload's batch
        {"name": "train_b8192", "kind": "train", "batch": 8192, "steps": 32},
        # a layered, lossy shot on 0.1 m cells
        {"name": "fdtd_281x201", "kind": "fdtd", "range_m": 26.0, "depth_m": 18.0, "spacing": 0.1, "steps": 500,
         "lossy": True},
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _logi(rng, lo, hi):
    return min(hi, max(lo, int(round(_log(rng, lo, hi)))))


def draw(rng):
    kind = rng.choice(["point", "default", "bank", "bank", "plan", "plan", "batch", "sobol", "impulse", "disp",
                       "predict", "train", "fdtd"])
    c = {"kind": kind}
    if kind == "point":
        c.update(layers=rng.randint(1, 6), nr=_logi(rng, 1, 64), rmax=round(_log(rng, 5, 64), 2),
                 freq=round(_log(rng, 5, 100), 3))
    elif kind == "default":
        fs, samples = rng.choice([(1000.0, 1024), (2000.0, 4096), (2000.0, 2048)])
        top = int(150.0 / (fs / samples))
        while True:
            c.update(layers=rng.randint(1, 4), nf=_logi(rng, 16, top), nr=_logi(rng, 4, 300),
                     rmax=round(_log(rng, 5, 40), 2), fs=fs, samples=samples)
            if work(c)["flops"] <= 4e9:  # a pass of no more than the loam bank's time
                break
    elif kind in ("bank", "plan"):
        big = 2048 * 16384 * 11
        while True:
            c.update(layers=rng.randint(1, 12), nf=_logi(rng, 16, 2048), nr=_logi(rng, 9, 1024),
                     nk=_logi(rng, 512, 16384), split=rng.random() < 0.5)
            if c["nf"] * c["nk"] * c["layers"] <= big:
                break
    elif kind == "batch":
        c.update(soils=_logi(rng, 3, 64), nr=_logi(rng, 16, 256), nk=_logi(rng, 2048, 8192),
                 split=rng.random() < 0.5)
    elif kind == "sobol":
        c.update(soils=_logi(rng, 8, 256))
    elif kind == "impulse":
        samples = rng.choice([256, 1024, 2048, 4096])
        c.update(count=_logi(rng, 2, 1024), samples=samples, nq=_logi(rng, 1, 8192),
                 length=_logi(rng, samples // 8, samples))
        c["nq"] = min(c["nq"], 8192 * 1024 // c["length"])
    elif kind == "disp":
        c.update(layers=rng.randint(2, 11), nf=_logi(rng, 1, 512), fmax=round(_log(rng, 30, 200), 2))
    elif kind == "predict":
        nr = rng.choice([1, 1, 3, 16])
        c.update(soils=_logi(rng, 1, 2048 // nr), nr=nr)
    elif kind == "train":
        c.update(batch=128 * _logi(rng, 8, 64), steps=rng.randint(4, 32))
    else:
        sp = round(_log(rng, 0.1, 0.4), 3)
        c.update(range_m=round(rng.uniform(8, 26), 1), depth_m=round(rng.uniform(6, 18), 1), spacing=sp,
                 steps=_logi(rng, 50, 500), lossy=rng.random() < 0.5)
    return c


# ------------------------------------------------------------------ inputs --

def _rng(case, seed):
    return np.random.default_rng([int(seed) & 0x7FFFFFFF, sum(ord(ch) for ch in case["kind"])])


def _graded(n, rng, top=120.0, bottom=600.0, h=0.8):
    """n stack entries as [thickness, Vp, Vs, density, Qs, Qp], Vs rising with depth."""
    rows = []
    for i in range(n):
        x = i / max(n - 1, 1)
        vs = (top + (bottom - top) * x) * rng.uniform(0.95, 1.05)
        qs = (10 + 50 * x) * rng.uniform(0.95, 1.05)
        rows.append([h * rng.uniform(0.9, 1.1) if i < n - 1 else 0.0, 2 * vs, vs, 1600 + 500 * x, qs, 2 * qs])
    return rows


def _uneven(nl, nf, rng):
    vs = np.exp(rng.uniform(math.log(80), math.log(600), nl))
    ratio, rho, qs = rng.uniform(1.7, 3.0, nl), rng.uniform(1500, 2200, nl), rng.uniform(10, 60, nl)
    h = np.exp(rng.uniform(math.log(0.2), math.log(5.0), nl))
    rows = [[float(h[i]) if i < nl - 1 else 0.0, float(vs[i] * ratio[i]), float(vs[i]), float(rho[i]), float(qs[i]),
             float(2 * qs[i])] for i in range(nl)]
    return rows, np.arange(1, nf + 1) * FS / (2 * nf)


def _soil(case, seed):
    """The soil(s), frequencies, ranges and grid of an f-k case."""
    rng, kind = _rng(case, seed), case["kind"]
    if kind in ("point", "default"):
        n = case["layers"]
        if n == 1:
            rows = [[0.0, 500.0 * rng.uniform(0.97, 1.03), 200.0 * rng.uniform(0.97, 1.03), 1700.0, 25.0, 0.0]]
        else:
            rows = _graded(n, rng, 160.0, 400.0, 1.2)
            rows = [r[:5] + [0.0] for r in rows]
        if kind == "point":
            ranges = np.array([case["rmax"] * 0.5]) if case["nr"] == 1 else np.geomspace(2.0, case["rmax"], case["nr"])
            return [rows], [np.array([case["freq"] * rng.uniform(0.97, 1.03)])], ranges, (0, 0.0), 0.0
        ranges = 1.0 + (case["rmax"] - 1.0) * np.arange(case["nr"]) / max(case["nr"] - 1, 1)
        freqs = np.arange(1, case["nf"] + 1) * case["fs"] / case["samples"]
        return [rows], [freqs], ranges, (0, 0.0), 0.0
    if kind in ("bank", "plan"):
        n, nf = case["layers"], case["nf"]
        rows = _graded(n, rng, 150.0, 400.0, 1.0) if n <= 3 else _graded(n, rng)
        vmin = 0.95 * min(150.0 if n <= 3 else 120.0, 400.0)
        freqs = np.arange(1, nf + 1) * FS / (2 * nf)
        ranges = np.arange(1, case["nr"] + 1) * (0.5 if case["nr"] > 128 else 1.0)
        kmax = max(2.5 * 2 * math.pi * 500.0 / vmin, 40 / ranges[0])
        return [rows], [freqs], ranges, (case["nk"], kmax), math.pi * FS / (2 * nf)
    if kind == "batch":
        sizes = np.random.default_rng(case["soils"])  # the same layer and bin counts for every seed
        soils = [_uneven(int(sizes.integers(2, 13)), int(sizes.integers(256, 2049)), rng) for _ in range(case["soils"])]
        return ([s for s, _ in soils], [f for _, f in soils], np.arange(1, case["nr"] + 1, dtype=np.float64),
                (case["nk"], KMAX_SOILS), 1.5)
    raise ValueError(kind)


def _stack(rows):
    return gfk.Stack([gfk.Layer(*r) for r in rows])


class _Device:
    """A plan's result buffer as an array that torch can look at; the plan lives as long as the view."""

    def __init__(self, plan, shape):
        self.plan, ptr = plan, plan.result_device_ptr()
        self.__cuda_array_interface__ = {"shape": shape, "typestr": "<f8", "data": (int(ptr), False), "version": 3}


def _view(plan, shape):
    return torch.as_tensor(_Device(plan, shape), device="cuda")


def _bank_payload(case, rng):
    """A bank's float32 payload: decaying, dispersing waves with a resonance."""
    count, bins = case["count"], case["samples"] // 2 + 1
    r = torch.linspace(1.0, 1.0 + 0.5 * (count - 1), count, dtype=torch.float64, device="cuda")[:, None]
    f = torch.arange(bins, dtype=torch.float64, device="cuda")[None, :] * FS / case["samples"]
    c = (120 + 80 * rng.uniform()) * (1 + 0.6 / (1 + (f / 25) ** 2))
    a = torch.exp(-2 * math.pi * f * r / (2 * 30 * c)) / torch.sqrt(r) * 1e-9 * (1 + rng.uniform() / (1 + (f / 40 - 1) ** 2))
    ph = -2 * math.pi * f * r / c
    out = torch.stack([a * torch.cos(ph), a * torch.sin(ph)], dim=2)
    out[:, 0] = 0.0
    return out.to(torch.float32).cpu().numpy()


def _sensor(case):
    s = 2j * np.pi * np.arange(case["samples"] // 2 + 1) * FS / case["samples"]
    w0 = 2 * np.pi * 10.0
    return 28.8 * s * s / (s * s + 1.4 * w0 * s + w0 * w0)


# the surrogate's soil family: (low, high, log-uniform) of its 11 scalars
FAMILY = [(80, 600, 1), (1.7, 3.0, 0), (10, 60, 0), (0.2, 5.0, 1), (80, 600, 1), (1.7, 3.0, 0), (10, 60, 0),
          (0.2, 5.0, 1), (80, 600, 1), (0.2, 5.0, 1), (80, 600, 1)]
WIDTH, NIN, NFOURIER = 512, 128, 47
SCALES = (1.0, 64.0, FS / 1024, 500.0)       # range and frequency domain
MEAN_STD = (-22.0, 2.5, 0.0045, 0.0005)      # of log|G| and the phase slowness


def _network(seed):
    """Network parameters in the flat order the package takes, and Fourier frequencies."""
    g = torch.Generator(device="cpu").manual_seed(int(seed))
    parts, fan = [], [NIN] + [WIDTH] * 5
    for l in range(6):
        out = WIDTH if l < 5 else 2
        b = 1 / math.sqrt(fan[l])
        parts += [(torch.rand(out * fan[l], generator=g) * 2 - 1) * b * (1.6 if l < 5 else 1.0),
                  (torch.rand(out, generator=g) * 2 - 1) * b]
    return torch.cat(parts).numpy(), (torch.randn(NFOURIER, 2, generator=g) * 8.0).numpy()


def _family(n, rng):
    u = rng.random((n, len(FAMILY)))
    out = np.empty_like(u)
    for j, (lo, hi, log) in enumerate(FAMILY):
        out[:, j] = np.exp(np.log(lo) + u[:, j] * (np.log(hi) - np.log(lo))) if log else lo + u[:, j] * (hi - lo)
    return out


def _predict_points(case):
    freqs = np.arange(1, 513) * FS / 1024
    return np.array([10.0]) if case["nr"] == 1 else np.linspace(2.0, 60.0, case["nr"]), freqs


SOBOL = [(80, 600, 1), (1.7, 3.0, 0), (10, 60, 0), (80, 600, 1), (1.7, 3.0, 0), (10, 60, 0), (0.2, 5.0, 1), (80, 600, 1)]


def _sobol_params(case, seed):
    u = _rng(case, seed).random((case["soils"], 8))
    out = np.empty_like(u)
    for j, (lo, hi, log) in enumerate(SOBOL):
        out[:, j] = np.exp(np.log(lo) + u[:, j] * (np.log(hi) - np.log(lo))) if log else lo + u[:, j] * (hi - lo)
    return out


def _fdtd_stack(case, seed):
    rng = _rng(case, seed)
    return [(2.0, 350.0, 140.0 * rng.uniform(0.97, 1.03), 1600.0), (0.0, 800.0, 320.0 * rng.uniform(0.97, 1.03), 2000.0)]


def _fdtd_setup(case, seed):
    st = _fdtd_stack(case, seed)
    sls = (lambda w, root: ((root - 1 / 25) / w, (root + 1 / 25) / w))(2 * math.pi * 30, math.sqrt(1 + 1 / 625))
    return st, sls if case["lossy"] else None, [2.0, 4.0, 6.5]


def prepare(case, seed):
    kind, eng = case["kind"], gfk.default_engine()
    st = {"kind": kind, "case": case, "engine": eng}
    if kind in ("point", "default", "bank", "plan", "batch"):
        rows, freqs, ranges, (nk, kmax), wi = _soil(case, seed)
        if kind in ("point", "default"):
            st["medium"] = gfk.Medium(_stack(rows[0]))
            st["ranges"], st["freq"] = ranges, float(freqs[0][0])
            if kind == "default":
                st["header"] = gfk.Header(gfk.Provenance("gfk"), _stack(rows[0]), case["fs"], case["samples"],
                                          gfk.RangeGrid(float(ranges[0]), float(ranges[-1]), len(ranges)),
                                          "vertical_displacement", "m/N")
                st["max_freq"] = float(freqs[0][-1]) * (1 + 1e-9)
            return st
        kw = dict(formulation=gfk.DUNKIN, omega_imag=wi, quadrature=gfk.SPLIT_INT8 if case["split"] else gfk.PLAIN_FP64)
        opt = gfk.Integration(nk, 0.0, kmax)
        if kind == "bank":
            st.update(medium=gfk.Medium(_stack(rows[0]), **kw), ranges=ranges, freqs=freqs[0], opt=opt)
            return st
        if kind == "plan":
            plan = gfk.Plan(gfk.Medium(_stack(rows[0]), **kw), ranges, freqs[0], opt)
        else:
            lay = np.array([r for s in rows for r in s])
            plan = gfk.Batch.from_layers(lay, [len(s) for s in rows], None, ranges, opt,
                                         (gfk.DUNKIN, kw["quadrature"], wi), freqs_per_medium=freqs)
            plan.use_graph()
        st.update(plan=plan, out=_view(plan, (sum(map(len, freqs)), len(ranges), 2)))
    elif kind == "sobol":
        st.update(params=_sobol_params(case, seed), setup=gfk.sobol.TraceSetup())
    elif kind == "impulse":
        rng = _rng(case, seed)
        top = 1.0 + 0.5 * (case["count"] - 1)
        h = gfk.Header(gfk.Provenance("gfk"), gfk.uniform(500.0, 200.0, 1700.0, 25.0), FS, case["samples"],
                       gfk.RangeGrid(1.0, top, case["count"]), "vertical_displacement", "m/N")
        st["bank"] = gfk.Bank(h, _bank_payload(case, rng)).device()
        st["q"] = rng.uniform(1.0, top, case["nq"])
        st["sensor"] = _sensor(case)
        st["out"] = torch.empty((case["nq"], case["length"]), dtype=torch.float64, device="cuda")
    elif kind == "disp":
        rng = _rng(case, seed)
        st["stack"] = _stack(_graded(case["layers"], rng))
        st["freqs"] = np.linspace(2.0, case["fmax"], case["nf"]) * rng.uniform(0.99, 1.0)
    elif kind == "predict":
        net = gfk.surrogate.Net(gfk.surrogate.NetConfig(batch=1024))
        p, four = _network(seed)
        net.set_params(p)
        net.set_fourier(four)
        net.set_scales(*SCALES, MEAN_STD)
        ranges, freqs = _predict_points(case)
        st.update(net=net, params=_family(case["soils"], _rng(case, seed)), ranges=ranges, freqs=freqs,
                  out=torch.empty((case["soils"], len(freqs), len(ranges), 2), dtype=torch.float64, device="cuda"))
    elif kind == "train":
        ds = gfk.surrogate.Dataset(_family(16, _rng(case, seed))).fill()
        net = gfk.surrogate.Net(gfk.surrogate.NetConfig(batch=case["batch"], seed=int(seed) % 100003))
        net.scales_from(ds)
        st.update(ds=ds, net=net, soils=np.arange(16, dtype=np.int32))
    elif kind == "fdtd":
        rows, sls, ranges = _fdtd_setup(case, seed)
        md = gfk.fdtd.Model(gfk.Stack([gfk.Layer(h, vp, vs, rho, 0, 0) for h, vp, vs, rho in rows]),
                            relax=gfk.SLS(*sls) if sls else None, ref_freq=30, max_range=case["range_m"],
                            depth=case["depth_m"], spacing=case["spacing"], dominant_freq=25)
        dt = md.grid()[0]
        st["shot"] = gfk.fdtd.Shot(md, gfk.fdtd.ricker(1000.0, 25.0, dt, case["steps"]), ranges, case["steps"])
    return st


# --------------------------------------------------------------------- run --

def run(state):
    kind, case = state["kind"], state["case"]
    if kind == "point":
        return state["medium"].vertical_displacement_multi(state["ranges"], state["freq"])
    if kind == "default":
        return gfk.build_bank(state["medium"], state["header"], state["max_freq"], check_range_sampling=False)[0].data
    if kind == "bank":
        return state["medium"].bank_spectra(state["ranges"], state["freqs"], state["opt"])[0]
    if kind in ("plan", "batch"):
        state["plan"].execute()
        return state["out"]
    if kind == "sobol":
        peak, centroid, _ = gfk.sobol.solve_metrics(state["params"], state["setup"], state["engine"])
        return peak, centroid
    if kind == "impulse":
        state["bank"].impulse_responses(state["q"], case["length"], state["sensor"], True,
                                        out_device_ptr=state["out"].data_ptr())
        return state["out"]
    if kind == "disp":
        modes = gfk.disp.modes_many(state["stack"], state["freqs"])
        curves = np.zeros((len(modes), 64))  # by mode, as a plot of them takes it
        for row, m in zip(curves, modes):
            row[:len(m)] = m
        return np.array([len(m) for m in modes]), curves
    if kind == "predict":
        state["net"].predict(state["params"], state["ranges"], state["freqs"], out_device_ptr=state["out"].data_ptr())
        return state["out"]
    if kind == "train":
        loss = state["net"].train(state["ds"], state["soils"], case["steps"])
        return loss, state["net"].params()
    res = gfk.fdtd.run(state["shot"])
    return np.array([t.vertical for t in res.traces])


# -------------------------------------------------------------------- work --

def _fk_work(points_layers, points, cells, nk_cells, out_bytes):
    # per (frequency, wavenumber): 700 FP64 flops a finite layer + 300; 4 a wavenumber of a cell
    return {"bytes": float(out_bytes), "flops": 700.0 * points_layers + 300.0 * points + 4.0 * nk_cells}


def work(case):
    kind = case["kind"]
    if kind in ("point", "default"):
        rows, freqs, ranges, _, _ = _soil(case, 1)
        nk = [_default_grid(rows[0], ranges, f)[1] for f in freqs[0]]
        nf, nr = len(freqs[0]), len(ranges)
        out = 16 * nr if kind == "point" else 8 * nr * (case["samples"] // 2 + 1)
        return _fk_work(sum(nk) * (len(rows[0]) - 1), sum(nk), nf * nr, sum(nk) * nr, out)
    if kind in ("bank", "plan", "batch"):
        rows, freqs, ranges, (nk, _), _ = _soil(case, 1)
        pts = sum(len(f) for f in freqs) * nk
        pl = sum(len(f) * (len(s) - 1) for s, f in zip(rows, freqs)) * nk
        cells = sum(len(f) for f in freqs) * len(ranges)
        return _fk_work(pl, pts, cells, pts * len(ranges), 16 * cells)
    if kind == "sobol":
        pts = case["soils"] * 512 * 8192
        return _fk_work(2 * pts, pts, case["soils"] * 512, pts, 16 * case["soils"])
    if kind == "impulse":
        bins, n = case["samples"] // 2 + 1, case["samples"]
        return {"bytes": 16.0 * min(case["count"], 2 * case["nq"]) * bins + 8.0 * case["nq"] * case["length"],
                "flops": case["nq"] * (2.5 * n * math.log2(n) + 60.0 * bins)}
    if kind == "disp":
        # the scan's 2001 evaluations of the secular function, about 300 flops a finite layer
        return {"bytes": 8.0 * case["nf"] * 8, "flops": case["nf"] * 2001.0 * (300.0 * (case["layers"] - 1) + 50)}
    macs = NIN * WIDTH + 4 * WIDTH * WIDTH + 2 * WIDTH
    if kind == "predict":
        rows = case["soils"] * 512.0 * case["nr"]
        return {"bytes": 16.0 * rows + 4.0 * macs, "flops": 2.0 * macs * rows}
    if kind == "train":
        # forward, gradient of activations and of weights; parameters and two moments read and written
        return {"bytes": case["steps"] * 24.0 * macs, "flops": case["steps"] * 2.0 * case["batch"] * (3.0 * macs - NIN * WIDTH)}
    nr, nz = int(case["range_m"] / case["spacing"]) + 21, int(case["depth_m"] / case["spacing"]) + 21
    fields = 10 if case["lossy"] else 6
    return {"bytes": case["steps"] * 16.0 * fields * nr * nz, "flops": case["steps"] * 80.0 * nr * nz}


# ------------------------------------------------------------------- exact --

def _default_grid(rows, ranges, f):
    slow = min(r[2] for r in rows)
    kb = 2 * math.pi * f / slow
    kmax = max(30 * kb, 40 / min(ranges))
    dk = min(2 * math.pi / (8 * max(ranges)), kb / (2 * rows[-1][4]) / 4)
    return kmax, max(64, math.ceil(kmax / dk))


def _velocity(v, q, f, wi):
    """Kjartansson constant-Q velocity at 2 pi f - i wi, reference 30 Hz; f: tensor [nf, 1]."""
    gam = math.atan(1 / q) / math.pi
    z = 1j * (2 * math.pi * f - 1j * wi) / (2 * math.pi * 30.0)
    return v * math.cos(math.pi * gam / 2) * torch.exp(gam * torch.log(z))


def _exact_u(rows, f, wi, k):
    """Surface displacement per newton at frequencies f [nf, 1] and wavenumbers
    k [nf or 1, nk]: the decaying half-space minors carried to the surface, in
    each layer's basis (pd, (sd - rb pd)/eb, pu, (su + rb pu)/eb), where the
    layer's exponential is upper triangular and bounded."""
    mu_ref = max(r[3] * r[2] ** 2 for r in rows)
    c2 = (2 * math.pi * f - 1j * wi) ** 2 / k ** 2
    m = None
    for h, vp, vs, rho, qs, qp in reversed(rows):
        a2 = _velocity(vp, qp if qp > 0 else 2.25 * qs, f, wi) ** 2
        b2 = _velocity(vs, qs, f, wi) ** 2
        ea, eb, kap, mu = c2 / a2, c2 / b2, b2 / a2, rho * b2 / mu_ref
        ra, rb = torch.sqrt(1 - ea), torch.sqrt(1 - eb)
        A, B = 1 / (1 + ra), 1 / (1 + rb)
        u1, d = kap * A + ra * B, B - kap * A  # (1 - ra rb)/eb, (ra - rb)/eb
        x2, s = 2 * u1 - 1, 2 - eb             # (1 + rb^2 - 2 ra rb)/eb, 1 + rb^2
        if m is None:
            m = [-u1, -mu * x2, mu * rb, -mu * ra, mu * mu * (4 * u1 - 4 + eb)]
            continue
        z = k * h
        Eb = torch.exp(-rb * z)
        em = torch.expm1(-d * eb * z)  # exp(-ra z)/exp(-rb z) - 1
        Ea, W = Eb * (1 + em), -rb * Eb * em / eb
        g3, g2 = mu * rb, mu * ra  # determinants of the blocks on (u_x, s_z) and (u_z, s_x)
        # minors in the two blocks' bases: adj(B03) V adj(B12)^T
        t00, t01 = u1 * m[1] - mu * x2 * m[0], ra * m[1] - 2 * g2 * m[0]
        t10, t11 = -(mu * x2 * m[1] + u1 * m[4]), -(2 * g2 * m[1] + ra * m[4])
        v03, v12 = g2 * m[2], g3 * m[3]
        v01, v02, v13, v23 = g3 * t00, g3 * t01, mu * s * t00 - t10, mu * s * t01 - t11
        y0, y5 = v02 - v13 + v03 - v12, v02 - v13 - v03 + v12
        y1, y2, y3, y4 = 2 * v01, v02 + v13 - v03 - v12, -(v02 + v13 + v03 + v12), -2 * v23
        # through the layer: [[Eb, -W], [0, Ea]] Y [[Ea, -W], [0, Eb]]^T, and 1, (Ea Eb)^2 outside
        p0, p1, p2, p3 = Eb * y1 - W * y3, Eb * y2 - W * y4, Ea * y3, Ea * y4
        z1, z2, z3, z4, z5 = Ea * p0 - W * p1, Eb * p1, Ea * p2 - W * p3, Eb * p3, (Ea * Eb) ** 2 * y5
        w01, w23 = 2 * z1, -2 * z4
        w02, w13 = y0 + z5 + z2 - z3, z2 - z3 - y0 - z5
        w03, w12 = y0 - z5 - z2 - z3, -(y0 - z5 + z2 + z3)
        U00, U01, U11 = ra * w01 - u1 * w02, 2 * g2 * w01 - mu * x2 * w02, mu * x2 * w23 - 2 * g2 * w13
        m = [U00, U01, g3 * w03, g2 * w12, -(mu * s * U01 + g3 * U11)]
        big = torch.stack([x.abs() for x in m]).amax(0)
        m = [x / big for x in m]
    return m[3] / (2 * math.pi * mu_ref * k * m[4])


def _j0(x):
    """Bessel J0: the midpoint rule on (1/pi) int cos(x sin t) dt below 25 (error
    J_64(x)), Hankel's asymptotic series above."""
    out, small = torch.empty_like(x), x < 25
    xs, xl = x[small], x[~small]
    out[small] = sum(torch.cos(xs * math.sin((j + 0.5) * math.pi / 32)) for j in range(16)) / 16
    P, Q, a, inv, p = torch.ones_like(xl), torch.zeros_like(xl), 1.0, 1 / xl, torch.ones_like(xl)
    for n in range(1, 25):
        a *= -((2 * n - 1) ** 2) / (8.0 * n)
        p = p * inv
        term = a * p if (n // 2) % 2 == 0 else -a * p
        P, Q = (P + term, Q) if n % 2 == 0 else (P, Q + term)
    s, c = torch.sin(xl), torch.cos(xl)
    out[~small] = torch.sqrt(inv / math.pi) * (P * (c + s) - Q * (s - c))
    return out


def _exact_rows(rows, freqs, wi, ranges, grid):
    """G [nf, nr] in complex128: the static-subtracted wavenumber sum."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    r = torch.as_tensor(np.asarray(ranges, dtype=np.float64), device=dev)
    slow, rmin = min(x[2] for x in rows), float(min(ranges))
    out = torch.zeros(len(freqs), len(r), dtype=torch.complex128, device=dev)
    shared = grid[0] > 0

    def weights(kmax, n):
        k = torch.arange(1, n + 1, dtype=torch.float64, device=dev) * (kmax / n)
        w = _j0(k[:, None] * r[None, :]) * (kmax / n)
        w[-1] *= 0.5
        return k, w

    if shared:
        k, w = weights(max(grid[1], 40 / rmin), grid[0])
    step = max(1, (1 << 21) // grid[0]) if shared else 1
    for a in range(0, len(freqs), step):
        f = torch.as_tensor(np.asarray(freqs[a:a + step], dtype=np.float64), device=dev)[:, None]
        if not shared:
            kmax, n = _default_grid(rows, ranges, float(f))
            k, w = weights(kmax, n)
        kf = torch.clamp(200 * 2 * math.pi * f / slow, min=400 / rmin)
        C = kf * _exact_u(rows, f, wi, kf)
        rem = k[None, :] * _exact_u(rows, f, wi, k[None, :]) - C
        G = torch.complex(rem.real @ w, rem.imag @ w)
        out[a:a + step] = G + C / r[None, :] - 0.5 * float(k[0]) * C
    return out


def _pairs(z):
    return torch.view_as_real(z)


def _exact_sobol(case, seed):
    setup = gfk.sobol.TraceSetup()
    S = torch.as_tensor(gfk.sobol.shaping(setup))[None, 1:]  # the source and sensor spectrum, an input here
    peak, cen = [], []
    f = np.arange(513) * FS / 1024
    band = torch.as_tensor((f >= 2) & (f <= 400))
    ft = torch.as_tensor(f)
    grow = torch.exp(setup.omega_imag * torch.arange(1024, dtype=torch.float64) / FS)
    for vs1, r1, q1, vs2, r2, q2, h1, vsh in _sobol_params(case, seed):
        rows = [[h1, r1 * vs1, vs1, 1700.0, q1, 2 * q1], [2.0, r2 * vs2, vs2, 1850.0, q2, 2 * q2],
                [0.0, 2 * vsh, vsh, 2000.0, 40.0, 80.0]]
        G = _exact_rows(rows, f[1:], setup.omega_imag, [10.0], (8192, KMAX_SOILS))[:, 0].cpu()
        Y = torch.zeros(513, dtype=torch.complex128)
        Y[1:] = G * S[0]
        y = torch.fft.irfft(Y, n=1024) * grow
        a = torch.fft.rfft(y).abs()[band]
        peak.append(float(y.abs().max()))
        cen.append(float((a * ft[band]).sum() / a.sum()))
    return np.array(peak), np.array(cen)


def _exact_impulse(case, seed):
    rng = _rng(case, seed)
    d = torch.as_tensor(_bank_payload(case, rng), device="cuda").double()
    top, count, n = 1.0 + 0.5 * (case["count"] - 1), case["count"], case["samples"]
    q = torch.as_tensor(rng.uniform(1.0, top, case["nq"]), device="cuda")
    z = torch.view_as_complex(d)
    lm, ang = torch.log(z.abs()), torch.angle(z)
    dp = torch.diff(ang, dim=0)
    turns = dp / (2 * math.pi)
    dp = dp - 2 * math.pi * torch.sign(turns) * torch.floor(turns.abs() + 0.5)
    ph = torch.cat([ang[:1], ang[:1] + torch.cumsum(dp, 0)])
    x = (q - 1.0) / ((top - 1.0) / (count - 1))
    lo = torch.clamp(torch.floor(x).long(), max=count - 2)
    fr = (x - lo)[:, None]
    f = torch.arange(n // 2 + 1, dtype=torch.float64, device="cuda") * FS / n
    from_f = 0.4 * FS
    taper = torch.where(f > from_f, 0.5 * (1 + torch.cos(math.pi * (f - from_f) / (0.5 * FS - from_f))), torch.ones_like(f))
    s = torch.as_tensor(_sensor(case), device="cuda") * (2j * math.pi * f) * taper
    out = torch.empty((case["nq"], case["length"]), dtype=torch.float64, device="cuda")
    for a in range(0, case["nq"], 512):
        l, t = lo[a:a + 512], fr[a:a + 512]
        H = torch.exp(torch.complex(lm[l] + t * (lm[l + 1] - lm[l]), ph[l] + t * (ph[l + 1] - ph[l]))) * s
        gone = ~torch.isfinite(lm[l] + lm[l + 1])  # a float32 zero at either end answers zero
        H[gone] = 0.0
        out[a:a + 512] = torch.fft.irfft(H, n=n)[:, :case["length"]]
    return out


def _exact_disp(case, seed):
    rng = _rng(case, seed)
    rows = _graded(case["layers"], rng)
    freqs = torch.as_tensor(np.linspace(2.0, case["fmax"], case["nf"]) * rng.uniform(0.99, 1.0), device="cuda")
    mu_ref = max(r[3] * r[2] ** 2 for r in rows)
    pairs = [(0, 1), (0, 2), (0, 3), (1, 2), (1, 3), (2, 3)]

    def secular(f, c):
        w, k = 2 * math.pi * f, 2 * math.pi * f / c
        m = torch.zeros(f.shape + (6,), dtype=torch.float64, device=f.device)
        m[..., 0] = 1
        for h, vp, vs, rho, _, _ in rows[:-1]:
            mu = rho * vs * vs
            lam = rho * vp * vp - 2 * mu
            l2, rc = lam + 2 * mu, rho * c * c
            M = torch.zeros(f.shape + (4, 4), dtype=torch.float64, device=f.device)
            M[..., 0, 1], M[..., 0, 2], M[..., 1, 0], M[..., 1, 3] = -1, mu_ref / mu, lam / l2, mu_ref / l2
            M[..., 2, 0], M[..., 2, 3] = (4 * mu * (lam + mu) / l2 - rc) / mu_ref, -lam / l2
            M[..., 3, 1], M[..., 3, 2] = -rc / mu_ref, 1
            grow = torch.sqrt(torch.clamp(1 - c * c / (vp * vp), min=0))
            P = torch.linalg.matrix_exp((M - grow[..., None, None] * torch.eye(4, dtype=torch.float64, device=f.device)) * (k * h)[..., None, None])
            C = torch.stack([torch.stack([P[..., i, a] * P[..., j, b] - P[..., i, b] * P[..., j, a] for a, b in pairs], -1)
                             for i, j in pairs], -2)
            m = (C @ m[..., None])[..., 0]
            m = m / m.abs().amax(-1, keepdim=True)
        _, vp, vs, rho, _, _ = rows[-1]
        mu, rc = rho * vs * vs, rho * c * c
        a, b = torch.sqrt(torch.clamp(1 - c * c / (vp * vp), min=0)), torch.sqrt(torch.clamp(1 - c * c / (vs * vs), min=0))
        one = torch.ones_like(a)
        p = [one, -a, -2 * mu / mu_ref * a, (2 * mu - rc) / mu_ref]
        s = [b, -one, (rc - 2 * mu) / mu_ref, 2 * mu / mu_ref * b]
        e = [p[i] * s[j] - p[j] * s[i] for i, j in pairs]
        return sum(g * m[..., i] * e[5 - i] for i, g in enumerate([1, -1, 1, 1, -1, 1]))

    lo, hi = 0.85 * min(r[2] for r in rows), rows[-1][2] * (1 - 1e-9)
    grid = lo + torch.arange(2001, dtype=torch.float64, device="cuda") * ((hi - lo) / 2000)
    vals = torch.cat([secular(f.expand(2001)[None], grid[None]) for f in freqs])
    fi, ci = torch.nonzero(vals[:, :-1] * vals[:, 1:] < 0, as_tuple=True)
    a, b, fa, f = grid[ci], grid[ci + 1], vals[fi, ci], freqs[fi]
    for _ in range(60):
        mid = 0.5 * (a + b)
        v = secular(f, mid)
        left = fa * v < 0
        a, fa, b = torch.where(left, a, mid), torch.where(left, fa, v), torch.where(left, mid, b)
    counts = torch.bincount(fi, minlength=len(freqs)).cpu().numpy()
    fi, roots, curves = fi.cpu().numpy(), (0.5 * (a + b)).cpu().numpy(), np.zeros((len(freqs), 64))
    for i in range(len(freqs)):
        curves[i, :counts[i]] = roots[fi == i]
    return counts, curves


def _exact_predict(case, seed):
    """The network with its BF16 weights and 64-bit activations."""
    flat, four = _network(seed)
    p = _family(case["soils"], _rng(case, seed))
    ranges, freqs = _predict_points(case)
    dev, t = "cuda", lambda x: torch.as_tensor(x, dtype=torch.float64, device="cuda")
    sc = np.stack([2 * (np.log(p[:, j] / lo) / np.log(hi / lo)) - 1 if log else 2 * (p[:, j] - lo) / (hi - lo) - 1
                   for j, (lo, hi, log) in enumerate(FAMILY)], 1)
    vs1, r1, _, h1, vs2, r2, _, h2, vs3, h3, _ = p.T
    tt = np.stack([h1 / vs1, h2 / vs2, h3 / vs3, h1 / (r1 * vs1), h2 / (r2 * vs2), h3 / (2 * vs3)], 1)
    sc, tt, fr, rg, fo = t(sc), t(tt), t(freqs), t(ranges), t(four)
    W, off, fan = [], 0, [NIN] + [WIDTH] * 5
    flat = torch.as_tensor(flat, device=dev)
    for l in range(6):
        o = WIDTH if l < 5 else 2
        w = flat[off:off + o * fan[l]].reshape(o, fan[l])
        off += o * fan[l]
        W.append(((w.bfloat16() if l < 5 else w).double(), flat[off:off + o].double()))
        off += o
    out = torch.empty((case["soils"], len(freqs), len(ranges)), dtype=torch.complex128, device=dev)
    r_lo, r_hi, f_lo, f_hi = SCALES
    step = max(1, (1 << 18) // (len(freqs) * len(ranges)))
    for a in range(0, case["soils"], step):
        s, T = sc[a:a + step], tt[a:a + step]
        shape = (len(s), len(fr), len(rg))
        f, r = fr[None, :, None].expand(shape), rg[None, None, :].expand(shape)
        ur, uf = (r - r_lo) / (r_hi - r_lo), (f - f_lo) / (f_hi - f_lo)
        X = torch.zeros(shape + (NIN,), dtype=torch.float64, device=dev)
        X[..., :11] = s[:, None, None, :]
        X[..., 11], X[..., 12] = 2 * ur - 1, 2 * uf - 1
        X[..., 13] = 2 * torch.log(r / r_lo) / math.log(r_hi / r_lo) - 1
        X[..., 14] = 2 * torch.log(f / f_lo) / math.log(f_hi / f_lo) - 1
        ft = f[..., None] * T[:, None, None, :]
        X[..., 16:28:2], X[..., 17:28:2] = torch.sin(2 * math.pi * ft), torch.cos(2 * math.pi * ft)
        X[..., 28:34] = torch.clamp((torch.log(ft) + 2) / 3, -2, 2)
        g = 2 * math.pi * (fo[:, 0] * ur[..., None] + fo[:, 1] * uf[..., None])
        X[..., 34::2], X[..., 35::2] = torch.sin(g), torch.cos(g)
        y = X.reshape(-1, NIN)
        for w, b in W[:5]:
            y = torch.nn.functional.silu(y @ w.T + b)
        y = (y @ W[5][0].T + W[5][1]).reshape(shape + (2,))
        t0, t1 = y[..., 0] * MEAN_STD[1] + MEAN_STD[0], y[..., 1] * MEAN_STD[3] + MEAN_STD[2]
        out[a:a + step] = torch.exp(torch.complex(t0, -t1 * 2 * math.pi * f * r))
    return _pairs(out)


def _exact_fdtd(case, seed):
    """The axisymmetric velocity-stress scheme with C-PML and one relaxation, in numpy."""
    st, sls, ranges = _fdtd_setup(case, seed)
    h, steps, pml = case["spacing"], case["steps"], 20
    mod = (lambda f: (1 + 2j * math.pi * f * sls[1]) / (1 + 2j * math.pi * f * sls[0])) if sls else None
    low = (1 / np.sqrt(mod(30.0))).real if sls else 1.0
    stiff = sls[1] / sls[0] if sls else 1.0
    nr, nz = int(round(case["range_m"] / h)) + 1 + pml, int(round(case["depth_m"] / h)) + 1 + pml
    vmax = max(l[1] for l in st) * low * math.sqrt(stiff)
    dt = 0.5 * h / (vmax * math.sqrt(2))
    rho, lam, mu = np.empty(nz), np.empty(nz), np.empty(nz)
    for j in range(nz):
        _, vp, vs, r = st[0] if j * h < st[0][0] else st[1]
        mp, ms = r * (vp * low) ** 2 * stiff, r * (vs * low) ** 2 * stiff
        rho[j], lam[j], mu[j] = r, mp - 2 * ms, ms
    nxt = np.minimum(np.arange(nz) + 1, nz - 1)
    rhoz, muz = 0.5 * (rho + rho[nxt]), 2 * mu * mu[nxt] / (mu + mu[nxt])

    def profile(n, offset, inner):
        thick = pml * h
        s = (np.arange(n) + offset) * h - inner
        x = np.minimum(s / thick, 1.0)
        d, al = -3 * vmax * math.log(1e-4) / (2 * thick) * x * x, math.pi * 25.0 * (1 - x)
        b = np.where(s > 0, np.exp(-(d + al) * dt), 1.0)
        return np.where(s > 0, d * (b - 1) / np.where(d + al > 0, d + al, 1.0), 0.0), b, (s > 0).astype(float)

    Ri, Rh = profile(nr, 0.0, case["range_m"]), profile(nr, 0.5, case["range_m"])
    Zi, Zh = ([p[:, None] for p in profile(nz, o, case["depth_m"])] for o in (0.0, 0.5))
    psi = {}

    def damp(name, p, d):
        psi[name] = p[1] * psi.get(name, 0.0) + p[0] * d
        return d + p[2] * psi[name]

    if sls:
        kappa, den = (stiff - 1) / stiff, 1 + dt / (2 * sls[0])
        decay, drive = (1 - dt / (2 * sls[0])) / den, dt * kappa / sls[0] / den
    mem = {}

    def rate(name, e):
        if not sls:
            return e
        old = mem.get(name, 0.0)
        mem[name] = decay * old - drive * e
        return e + 0.5 * (old + mem[name])

    vr, vz, trr, tqq, tzz, trz = (np.zeros((nz, nr)) for _ in range(6))
    rh, ri = (np.arange(nr) + 0.5) * h, np.arange(nr) * h
    ri[0] = 1.0
    lamc, muc, l2m = lam[:, None], mu[:, None], (lam + 2 * mu)[:, None]
    t = np.arange(steps) * dt - 1.5 / 25.0
    arg = (math.pi * 25.0) ** 2
    force = 1000.0 * (1 - 2 * arg * t * t) * np.exp(-arg * t * t)
    force = np.append(force, [0.0, 0.0])
    cols = [min(int(round(r / h)), nr - 2) for r in ranges]
    area, traces = math.pi * h * h / 4, np.zeros((len(cols), steps))

    def padded(a, z=nz, r=nr):
        out = np.zeros((z, r))
        out[:a.shape[0], :a.shape[1]] = a
        return out

    for n in range(steps):
        tzz[0, 0] = -force[n] / area
        # velocities, on [0, nz-1) x [0, nr-1)
        a = damp("a", Rh, padded((trr[:, 1:] - trr[:, :-1]) / h))
        up = np.vstack([-trz[:1], trz[:-1]])
        b = damp("b", Zi, (trz - up) / h)
        hoop = padded(0.5 * ((trr - tqq)[:, 1:] + (trr - tqq)[:, :-1]) / rh[:-1])
        c = damp("c", Zh, padded((tzz[1:] - tzz[:-1]) / h))
        left = np.hstack([-trz[:, :1], trz[:, :-1]])
        e = damp("d", Ri, (trz - left) / h) + 0.5 * (trz + left) / ri
        e[:, 0] = 4 * trz[:, 0] / h
        vr[:-1, :-1] += (dt / rho[:, None] * (a + b + hoop))[:-1, :-1]
        vz[:-1, :-1] += (dt / rhoz[:, None] * (c + e))[:-1, :-1]
        # surface velocity half a cell above the first row
        for q, i in enumerate(cols):
            g = 4 * vr[0, 0] / h if i == 0 else (vr[0, i] - vr[0, i - 1]) / h + 0.5 * (vr[0, i] + vr[0, i - 1]) / (i * h)
            traces[q, n] = vz[0, i] + 0.5 * h * lam[0] / (lam[0] + 2 * mu[0]) * g
        # stresses
        lft = np.hstack([-vr[:, :1], vr[:, :-1]])
        dvr, vrr = (vr - lft) / h, 0.5 * (vr + lft) / ri
        vrr[:, 0] = dvr[:, 0]
        dvr = damp("e", Ri, dvr)
        dvz = damp("f", Zi, (vz - np.vstack([vz[:1], vz[:-1]])) / h)
        applied = np.zeros(nr)
        applied[0] = (force[n + 1] - force[n]) / dt
        dvz[0] = (applied - lam[0] * (dvr[0] + vrr[0])) / l2m[0]
        trr += dt * rate("r", l2m * dvr + lamc * (vrr + dvz))
        tqq += dt * rate("q", lamc * (dvr + dvz) + l2m * vrr)
        tzz[1:] += dt * rate("z", lamc * (dvr + vrr) + l2m * dvz)[1:]
        s1 = damp("g", Rh, padded((vz[:, 1:] - vz[:, :-1]) / h))
        s2 = damp("h", Zh, padded((vr[1:] - vr[:-1]) / h))
        trz[:-1, :-1] += dt * rate("s", muz[:, None] * (s1 + s2))[:-1, :-1]
    return traces


def exact(case, seed):
    kind = case["kind"]
    if kind in ("point", "default", "bank", "plan", "batch"):
        rows, freqs, ranges, grid, wi = _soil(case, seed)
        G = torch.cat([_exact_rows(s, f, wi, ranges, grid) for s, f in zip(rows, freqs)])
        if kind == "point":
            return G[0].cpu().numpy()
        if kind == "bank":
            return G.cpu().numpy()
        if kind == "default":
            out = np.zeros((len(ranges), case["samples"] // 2 + 1, 2))
            out[:, 1:1 + len(freqs[0])] = _pairs(G.T.contiguous()).cpu().numpy()
            return out
        return _pairs(G)
    if kind == "sobol":
        return _exact_sobol(case, seed)
    if kind == "impulse":
        return _exact_impulse(case, seed)
    if kind == "disp":
        return _exact_disp(case, seed)
    if kind == "predict":
        return _exact_predict(case, seed)
    if kind == "fdtd":
        return _exact_fdtd(case, seed)
    return None  # train: each step's batch is drawn by the network's own generator
