"""Timed workloads of the engine: what its users run, from the smallest run to the largest.

Every case goes through the Python entry points (run_rewl, Engine, Batch, System).  Systems are
dipoles with random unit axes on simple cubic lattices (the benchmark's dense workload), on
lattices with missing sites (its mixed-precision workload) or at dilute random places (its
batched workload); the energy grid spans a multiple of sigma, the standard deviation of the
energy over random configurations; a power-of-two bin width is the largest below that spacing.

kinds of pass:
  run      run_rewl from geometry to fragments: engine creation (couplings, walker
           construction), the epochs up to max_mcs, the fragments and walker statistics.
  advance  a long run's next `epochs` epochs and the current fragments, on an engine that is
           already `warm` epochs into its run (the state a long production run is in).
  batch    many small single-window runs advanced together by one Batch.
  fields   local_fields: fields and energies of many configurations of one system.
"""
import math

import numpy as np

from replica_exchange_wang_landau_b200 import engine as E


def listed():
    return [
        # the quickest real call: the 2x2x2 lattice of the validation runs, one window, two walkers
        _case("cube_8_run", kind="run", nx=2, ny=2, nz=2, windows=1, walkers=2, bins=160, span=5.0, mcs=2000.0),
        # a small convergence study: two windows of two walkers, a bin width that is no power of two
        _case("cell_27_run", kind="run", nx=3, ny=3, nz=3, windows=2, walkers=2, bins=200, pow2=False, mcs=1000.0),
        # the adaptive-window pilot: the same run with pilot statistics switched on
        _case("pilot_343_run", kind="run", nx=7, ny=7, nz=7, windows=8, walkers=4, bins=400, collect=True, mcs=60.0,
              exchange_mcs=1.0),
        # the benchmark's dense shape as one whole call: 8x8x8, 16 windows x 8 walkers
        _case("dense_512_run", kind="run", nx=8, ny=8, nz=8, windows=16, walkers=8, bins=760, span=5.1, mcs=200.0,
              exchange_mcs=1.0),
        # the same shape in the middle of a long production run
        _case("dense_512_advance", kind="advance", nx=8, ny=8, nz=8, windows=16, walkers=8, bins=760, span=5.1,
              exchange_mcs=1.0, warm=400, epochs=96),
        # an odd lattice, rows that are no multiple of the padding, width no power of two
        _case("dense_990_run", kind="run", nx=9, ny=10, nz=11, windows=12, walkers=6, bins=777, pow2=False, mcs=40.0,
              exchange_mcs=1.0),
        # the mixed-precision shape (16x16x16 with 40% of the sites missing, slab, 32 x 8) in FP64 ...
        _case("slab_2458_fp64_advance", kind="advance", nx=16, ny=16, nz=16, removed=0.4, slab=True, windows=32,
              walkers=8, bins=900, exchange_mcs=1.0, warm=4, epochs=8),
        # ... and with FP32 couplings and the FP64 recompute after every MCS
        _case("slab_2458_fp32_advance", kind="advance", nx=16, ny=16, nz=16, removed=0.4, slab=True, windows=32,
              walkers=8, bins=900, precision="fp32", exchange_mcs=1.0, warm=4, epochs=8),
        # a cutoff system of the size the dense form serves too
        _case("csr_1000_run", kind="run", nx=10, ny=10, nz=10, cutoff=2.2, windows=8, walkers=8, bins=600, mcs=100.0,
              exchange_mcs=1.0),
        # the largest: 32x32x32, cutoff 3.0, 64 windows x 16 walkers, exchange every 0.05 MCS
        _case("csr_32768_advance", kind="advance", nx=32, ny=32, nz=32, cutoff=3.0, windows=64, walkers=16, bins=1000,
              exchange_mcs=0.05, warm=8, epochs=16),
        # training curves for the learned start: many dilute single-window systems side by side
        _case("batch_dilute_advance", kind="batch", instances=96, lo=64, hi=1024, walkers=2, bins=200,
              epoch_attempts=8192, warm=4, epochs=4),
        # energies of a set of stored configurations, as post-processing asks for them
        _case("fields_1000x256", kind="fields", nx=10, ny=10, nz=10, configurations=256),
    ]


_DEFAULTS = {
    "run": dict(nx=4, ny=4, nz=4, removed=0.0, slab=False, cutoff=0.0, precision="fp64", windows=1, walkers=2,
                bins=200, span=4.0, pow2=True, collect=False, exchange_mcs=10.0, mcs=100.0),
    "advance": dict(nx=4, ny=4, nz=4, removed=0.0, slab=False, cutoff=0.0, precision="fp64", windows=1, walkers=2,
                    bins=200, span=4.0, pow2=True, collect=False, exchange_mcs=1.0, warm=8, epochs=8),
    "batch": dict(instances=8, lo=16, hi=256, walkers=2, bins=200, epoch_attempts=8192, warm=4, epochs=4),
    "fields": dict(nx=6, ny=6, nz=6, configurations=16),
}


def _case(name, kind, **values):
    case = dict(_DEFAULTS[kind], kind=kind)
    case.update(values)
    if name:
        case["name"] = name
    return case


def _log_uniform(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    """One more case of the same ranges: lattices of 8 to 2500 sites (cutoff systems up to 32768),
    1 to 32 windows, 2 to 8 walkers each, every precision and option the listed cases use."""
    what = rng.choice(["dense", "dense", "dense", "dense", "csr", "csr", "pilot", "batch", "fields", "advance"])
    if what == "batch":
        lo = int(_log_uniform(rng, 16, 128))
        return _case(None, "batch", instances=rng.randint(8, 96), lo=lo, hi=lo + rng.randint(10, 1024 - lo),
                     walkers=rng.choice([1, 2, 2, 3]), epoch_attempts=rng.choice([1000, 4096, 8192]),
                     epochs=rng.randint(1, 4))
    n = _log_uniform(rng, 30, 30000) if what == "csr" else _log_uniform(rng, 8, 2500)
    side = n ** (1.0 / 3.0)
    nx = max(2, round(side * rng.uniform(0.8, 1.25)))
    ny = max(2, round(side * rng.uniform(0.8, 1.25)))
    nz = max(2, round(n / (nx * ny)))
    if what == "fields":
        return _case(None, "fields", nx=nx, ny=ny, nz=nz, configurations=max(1, int(_log_uniform(rng, 1, 300))))
    sites = nx * ny * nz
    windows = 1 if sites < 27 else rng.choice([1, 2, 3, 4, 8, 16] if sites < 200 else [1, 2, 4, 8, 16, 24, 32])
    values = dict(nx=nx, ny=ny, nz=nz, windows=windows, walkers=rng.randint(2, 8),
                  bins=rng.randint(max(100, 16 * windows), max(300, 30 * windows)), pow2=rng.random() < 0.6,
                  span=rng.uniform(3.0, 4.0))
    if what == "csr":
        values["cutoff"] = rng.choice([1.5, 2.2, 3.0])
        values["precision"] = rng.choice(["fp64", "fp64", "fp32"])
    elif what == "pilot":
        values["collect"] = True
    else:
        values["removed"] = rng.choice([0.0, 0.0, 0.0, 0.2, 0.4]) if sites > 100 else 0.0
        values["slab"] = rng.random() < 0.2
        values["precision"] = rng.choice(["fp64", "fp64", "fp64", "fp32", "bf16"])
    # attempts of all walkers together, so that a pass costs no more than the largest listed one
    chains = windows * values["walkers"]
    attempts = min(_log_uniform(rng, 1e4, 6e4), 6e6 / chains)
    if what == "advance":
        epochs = rng.randint(4, 16)
        return _case(None, "advance", exchange_mcs=attempts / epochs / sites, epochs=epochs, warm=8, **values)
    exchange = rng.choice([0.5, 1.0, 1.0, 10.0])
    return _case(None, "run", exchange_mcs=exchange, mcs=max(1.0, attempts / sites), **values)


# ---- systems --------------------------------------------------------------------------------


def _axes(rng, n):
    a = rng.standard_normal((n, 3))
    return a / np.sqrt((a * a).sum(axis=1, keepdims=True))


def _lattice(case, seed):
    """Random unit axes on a lattice (with `removed` of its sites missing), periodic in all
    directions or, for a slab, in two."""
    rng = np.random.default_rng(1000 + seed)
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    z, y, x = np.meshgrid(np.arange(nz), np.arange(ny), np.arange(nx), indexing="ij")
    pos = np.stack([x.ravel(), y.ravel(), z.ravel()], axis=1).astype(np.float64)
    removed = int(round(case["removed"] * len(pos)))
    if removed:
        pos = pos[np.sort(rng.permutation(len(pos))[removed:])]
    box = (float(nx), float(ny), 0.0 if case["slab"] else float(nz))
    return E.Geometry(pos, _axes(rng, len(pos)), box, True)


def _dilute(rng, n):
    """n sites at density about 0.5: lattice sites of a box twice as large, each moved a little."""
    side = int(math.ceil((2.0 * n) ** (1.0 / 3.0)))
    at = np.sort(rng.permutation(side ** 3)[:n])
    pos = np.stack([at % side, at // side % side, at // (side * side)], axis=1).astype(np.float64)
    pos += rng.uniform(-0.2, 0.2, pos.shape)
    return E.Geometry(pos, _axes(rng, n), (float(side),) * 3, True)


def _sigma(geometry, cutoff):
    """Standard deviation of the energy over random configurations: for independent random axes
    a pair at distance r adds (2/3) / r^6 on average; up to 600 sites are summed over."""
    pos = geometry.positions
    n = len(pos)
    some = pos[:: max(1, n // 600)]
    total = 0.0
    for p in some:
        d = pos - p
        for k in range(3):
            if geometry.box[k] > 0.0:
                d[:, k] -= geometry.box[k] * np.rint(d[:, k] / geometry.box[k])
        r2 = (d * d).sum(axis=1)
        r2 = r2[(r2 > 0.0) & ((r2 <= cutoff * cutoff) if cutoff > 0.0 else True)]
        total += float((1.0 / r2 ** 3).sum())
    return math.sqrt(0.5 * n * (2.0 / 3.0) * total / len(some))


def _config(case, geometry, seed):
    sigma = _sigma(geometry, case["cutoff"])
    bins = case["bins"]
    width = 2.0 * case["span"] * sigma / bins
    width = 2.0 ** math.floor(math.log2(width)) if case["pow2"] else round(width, 3)
    c = E.RunConfig(emin=-(bins // 2) * width, emax=(bins - bins // 2) * width, bin_width=width,
                    windows=case["windows"], walkers=case["walkers"], overlap=0.75, seed=seed + 1)
    c.wl = E.WlParameters(collect_window_statistics=case["collect"])
    c.check_interval_mcs = 1000.0 / geometry.size()  # the benchmark's check every 1000 attempts
    c.coupling_precision = case["precision"]
    c.exchange_interval_mcs = case["exchange_mcs"]
    c.max_mcs = case["mcs"] if case["kind"] == "run" else 0.0
    c.resolve_mcs(geometry.size())
    return c


def _spins(rng, count, n):
    return rng.integers(0, 2, size=(count, n)).astype(np.int8) * 2 - 1


# ---- one pass ---------------------------------------------------------------------------------


def prepare(case, seed):
    if case["kind"] == "fields":
        rng = np.random.default_rng(seed)
        geometry = _lattice(dict(case, removed=0.0, slab=False), seed)
        geometry.positions = geometry.positions + rng.uniform(-0.05, 0.05, geometry.positions.shape)
        return {"kind": "fields", "system": E.System(geometry), "spins": _spins(rng, case["configurations"],
                                                                                geometry.size())}
    if case["kind"] == "batch":
        rng = np.random.default_rng(seed)
        engines = []
        for k in range(case["instances"]):
            geometry = _dilute(rng, int(rng.integers(case["lo"], case["hi"] + 1)))
            sigma = _sigma(geometry, 0.0)
            width = 2.0 ** round(math.log2(8.0 * sigma / case["bins"]))
            half = case["bins"] // 2 * width
            c = E.RunConfig(emin=-half, emax=half, bin_width=width, windows=1, walkers=case["walkers"],
                            seed=seed * 1000 + k + 1)
            c.exchange_interval_uses_mcs = False
            c.exchange_interval_attempts = case["epoch_attempts"]
            c.max_mcs = 0.0
            c.resolve_mcs(geometry.size())
            e = E.Engine(E.System(geometry), c)
            e.set_launch(0, case["epochs"])
            engines.append(e)
        batch = E.Batch(engines)
        batch.run_epochs(case["warm"])
        return {"kind": "batch", "engines": engines, "batch": batch, "epochs": case["epochs"]}
    geometry = _lattice(case, seed)
    system = E.System(geometry, 1.0, case["cutoff"])
    config = _config(case, geometry, seed)
    if case["kind"] == "run":
        return {"kind": "run", "system": system, "config": config}
    engine = E.Engine(system, config)
    engine.run_epochs(case["warm"])
    return {"kind": "advance", "engine": engine, "epochs": case["epochs"], "collect": case["collect"]}


def _outputs(fragments, statistics):
    return {
        "log_g": np.stack([f.log_g for f in fragments]),
        "histogram": np.stack([f.histogram for f in fragments]),
        "standard_error": np.stack([f.standard_error for f in fragments]),
        "valid": np.stack([f.valid for f in fragments]),
        "energy": np.array([s["energy"] for s in statistics]),
        "factor": np.array([s["factor"] for s in statistics]),
        "counts": np.array([[s["attempted"], s["accepted"], s["active_bins"], s["minimum_histogram"],
                             s["round_trips"]] for s in statistics], dtype=np.int64),
    }


def run(state):
    kind = state["kind"]
    if kind == "run":
        r = E.run_rewl(state["system"], state["config"])
        out = _outputs(r.fragments, r.walker_statistics)
        out["exchanges"] = np.array([r.exchange_attempted, r.exchange_accepted, r.epochs], dtype=np.int64)
        if r.sampling_statistics:
            out["squared_displacement"] = np.stack([s.squared_energy_displacement for s in r.sampling_statistics])
            out["displacement_samples"] = np.stack([s.displacement_samples for s in r.sampling_statistics])
            out["representative_energy"] = np.array([e for e, _ in r.representatives])
            out["representative_spins"] = np.stack([s for _, s in r.representatives])
        return out
    if kind == "advance":
        e = state["engine"]
        e.run_epochs(state["epochs"])
        return _outputs(e.fragments(allow_empty=True), e.walker_statistics())
    if kind == "batch":
        state["batch"].run_epochs(state["epochs"])
        fragments = [e.fragment(0, allow_empty=True) for e in state["engines"]]
        return _outputs(fragments, [s for e in state["engines"] for s in e.walker_statistics()])
    fields, energies = state["system"].local_fields(state["spins"])
    return {"fields": fields, "energies": energies}


# ---- what a pass cannot do without ----------------------------------------------------------------


def work(case):
    """Bytes: the couplings and the walkers' state read once, the state and the fragments written
    once.  flops: per attempt the energy difference and the acceptance (about 10), per accepted
    flip (about 0.6 of them) a multiply and an add for every coupling of the flipped site."""
    if case["kind"] == "fields":
        n, k = case["nx"] * case["ny"] * case["nz"], case["configurations"]
        return {"bytes": n * 48 + k * n * 9 + k * 8, "flops": 2.0 * n * n * k}
    if case["kind"] == "batch":
        n = (case["lo"] + case["hi"]) / 2.0
        chains = case["instances"] * case["walkers"]
        attempts = float(case["epoch_attempts"]) * case["epochs"] * chains
        return {"bytes": case["instances"] * (n * n * 8 + case["bins"] * 25) + chains * (n * 18 + case["bins"] * 34),
                "flops": attempts * (10 + 0.6 * 2 * n)}
    n = case["nx"] * case["ny"] * case["nz"] * (1.0 - case["removed"])
    chains = case["windows"] * case["walkers"]
    size = {"fp64": 8, "fp32": 4, "bf16": 2}[case["precision"]]
    if case["cutoff"] > 0.0:
        z = min(n - 1, 4.19 * case["cutoff"] ** 3)
        couplings = n * z * (4 + size)
    else:
        z, couplings = n, n * n * size
    per_walker = case["mcs"] * n if case["kind"] == "run" else case["epochs"] * case["exchange_mcs"] * n
    return {"bytes": couplings + chains * (n * 18 + case["bins"] * 34) + case["windows"] * case["bins"] * 25,
            "flops": chains * per_walker * (10 + 0.6 * 2 * z)}


def exact(case, seed):
    """Fields and energies in 64 bits; a Markov chain's outputs have no such value."""
    if case["kind"] != "fields":
        return None
    state = prepare(case, seed)
    g, s = state["system"].geometry, state["spins"].astype(np.float64)
    n = g.size()
    box = np.asarray(g.box)
    fields = np.zeros(s.shape)
    for i in range(n):
        d = g.positions - g.positions[i]
        d -= box * np.rint(d / box)
        r2 = (d * d).sum(axis=1)
        r2[i] = 1.0
        r = np.sqrt(r2)
        ri = d / r[:, None]
        j = (g.axes @ g.axes[i] - 3.0 * (g.axes * ri).sum(axis=1) * (ri @ g.axes[i])) / (r2 * r)
        j[i] = 0.0
        fields[:, i] = s @ j
    return {"fields": fields, "energies": 0.5 * (s * fields).sum(axis=1)}
