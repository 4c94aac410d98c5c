"""The CSR sweep (csrc/sweep_csr.cu) where it runs, beyond 2048 sites: walker trajectories and run_rewl
(src/wang_landau.cpp:244-315, src/parallel.cpp:276-747) bit for bit against the oracle, for ELLPACK rows of 32,
64, 128 and 256 entries, FP64 and FP32 couplings, bin widths that are and are not powers of two, pilot
statistics, forced acceptance, the 1/t stage, a continued schedule and rejected draws.  (Smaller cutoff systems
run in the look-ahead sweep, so every case asserts the sweep.)"""
from __future__ import annotations

import dataclasses

import numpy as np
import pytest

from helpers import random_axes, results_equal, snapshots_equal
from test_gpu_rejected_draws import zero_draw_state
from replica_exchange_wang_landau_b200.engine import Engine, Geometry, RunConfig, System, run_rewl

pytestmark = pytest.mark.gpu

# 13^3 = 2197 sites: neighbours within 1.8, 2.2, 2.3, 2.5 and 3.5 lattice constants: 18, 32, 56, 80, 178
ROWS = {1.8: 32, 2.2: 32, 2.3: 64, 2.5: 128, 3.5: 256}


def _system(cutoff, seed=23, random=True):
    g = Geometry.simple_cubic(13, 13, 13, periodic=True)
    if random:
        g.axes = random_axes(g.size(), seed)
    return System(g, 1.0, cutoff)


def _config(width, precision="fp64", **kw):
    c = RunConfig(emin=-300 * width, emax=300 * width, bin_width=width, windows=2, walkers=2, **kw)
    c.coupling_precision = precision
    return c


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("width", [0.5, 0.6])
@pytest.mark.parametrize("cutoff", list(ROWS))
def test_trajectories(oracle, cutoff, width, precision):
    s = _system(cutoff)
    c = _config(width, precision, seed=31)
    c.resolve_mcs(s.size())
    with Engine(s, c) as e:
        assert e.sweep == "csr"
        for w in range(e.walkers):
            ow = oracle.walker(s, w, c.emin, c.emax, c.bin_width, e.window(w // c.walkers), c.wl, c.seed)
            assert snapshots_equal(e.snapshot(w), ow.snapshot()) == [], f"init of walker {w}"
            if precision == "fp32":
                ow.set_update_fp32(True)
            for rounds in range(2):
                e.run_attempts(w, 4001 + 311 * rounds)
                ow.run_attempts(4001 + 311 * rounds)
                assert snapshots_equal(e.snapshot(w), ow.snapshot()) == [], f"walker {w} round {rounds}"


RUNS = {
    "exchange": (2.3, dict(width=0.6, seed=41, exchange_interval_mcs=0.25, check_interval_mcs=1, max_mcs=8), {}),
    "exchange_fp32": (2.5, dict(width=0.5, precision="fp32", seed=42, exchange_interval_mcs=0.5, check_interval_mcs=1,
                                max_mcs=8), {}),
    "pilot": (2.5, dict(width=0.75, seed=44, exchange_interval_mcs=0.5, check_interval_mcs=1, max_mcs=8),
              dict(collect_window_statistics=True)),
    "pilot_wide_rows": (3.5, dict(width=0.5, seed=45, exchange_interval_mcs=0.5, check_interval_mcs=1, max_mcs=8),
                        dict(collect_window_statistics=True)),
}


@pytest.mark.parametrize("name", list(RUNS))
def test_runs(oracle, name):
    cutoff, kw, wl = RUNS[name]
    s = _system(cutoff)
    c = _config(**kw)
    for k, v in wl.items():
        setattr(c.wl, k, v)
    c.resolve_mcs(s.size())
    with Engine(s, c) as e:
        assert e.sweep == "csr"
    got = run_rewl(s, c)
    assert got.exchange_accepted > 0
    assert results_equal(got, oracle.run_rewl(s, c)) == []


@pytest.mark.parametrize("cutoff, width, precision", [(2.2, 16.0, "fp64"), (2.3, 17.0, "fp64"), (2.5, 16.0, "fp32"),
                                                      (3.5, 17.0, "fp64")])
def test_inverse_time_stage(oracle, cutoff, width, precision):
    """Bins so wide that all are visited within a few sweeps over the sites."""
    s = _system(cutoff)
    c = RunConfig(emin=-9 * width, emax=9 * width, bin_width=width, windows=2, walkers=2, seed=43, max_mcs=60,
                  exchange_interval_mcs=1, check_interval_mcs=2)
    c.coupling_precision = precision
    c.wl.minimum_visits, c.wl.final_factor = 1, 1e-4
    c.resolve_mcs(s.size())
    with Engine(s, c) as e:
        assert e.sweep == "csr"
    got, want = run_rewl(s, c), oracle.run_rewl(s, c)
    assert results_equal(got, want) == []
    assert all(0.0 < w["factor"] < 1e-3 for w in got.walker_statistics)


@pytest.mark.parametrize("width", [0.5, 0.6])
def test_forced_acceptance(oracle, width):
    s = _system(1.8, random=False)
    c = _config(width, seed=35, max_mcs=6, exchange_interval_mcs=0.5, check_interval_mcs=1)
    c.force_accept_after_uses_mcs = False
    c.wl.force_accept_after_attempts = 3
    c.resolve_mcs(s.size())
    with Engine(s, c) as e:
        assert e.sweep == "csr"
    got = run_rewl(s, c)
    assert got.forced_accepted > 0
    assert results_equal(got, oracle.run_rewl(s, c)) == []


@pytest.mark.parametrize("collect", [False, True])
@pytest.mark.parametrize("cutoff", [2.2, 2.3, 3.5])
def test_rejected_draws(oracle, cutoff, collect):
    """(2^64 - 2197) mod 2197 is not 0, so that a 0 draw is rejected as a site draw."""
    assert ((1 << 64) - 2197) % 2197 > 0
    s = _system(cutoff)
    c = _config(0.5, seed=51)
    c.wl.collect_window_statistics = collect
    c.resolve_mcs(s.size())
    with Engine(s, c) as e:
        assert e.sweep == "csr"
        for w in (0, 3):
            ow = oracle.walker(s, w, c.emin, c.emax, c.bin_width, e.window(w // c.walkers), c.wl, c.seed)
            for rounds, k in enumerate((0, 1, 2, 3, 6, 13, 40)):
                snap = dataclasses.replace(e.snapshot(w), rng_state=zero_draw_state(k, 100 * w + k))
                e.restore(w, snap)
                ow.restore(snap)
                e.run_attempts(w, 150 + 37 * rounds)
                ow.run_attempts(150 + 37 * rounds)
                assert snapshots_equal(e.snapshot(w), ow.snapshot()) == [], f"walker {w}, zero draw {k}"


@pytest.mark.parametrize("continue_schedule", [False, True])
@pytest.mark.parametrize("cutoff, width", [(2.2, 16.0), (2.5, 17.0)])
def test_warm_start(oracle, cutoff, width, continue_schedule):
    s = _system(cutoff)
    c = RunConfig(emin=-9 * width, emax=9 * width, bin_width=width, windows=2, walkers=2, seed=46, max_mcs=40,
                  exchange_interval_mcs=1, check_interval_mcs=2)
    c.wl.final_factor = 1e-6
    c.resolve_mcs(s.size())
    lg = -3.0 * np.linspace(-1.0, 1.0, c.bins()) ** 2
    with Engine(s, c) as e:
        assert e.sweep == "csr"
        e.warm_start(lg, 1e-3, continue_schedule=continue_schedule)
        e.run()
        got = e.result()
        assert all(e.snapshot(w).stage > 0 for w in range(e.walkers))  # the 1/t stage, or past it
    assert results_equal(got, oracle.run_rewl(s, c, warm_start=(lg, 1e-3, continue_schedule))) == []
