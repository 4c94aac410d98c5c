"""Pilot statistics in the look-ahead sweep (csrc/sweep_ahead.cu) where the fields of a block come later than its
entries: two walkers to an SM, and thousands of sites.  Runs with squared displacements, samples, round trips and
representatives, bit for bit against the CPU oracle."""
from __future__ import annotations

import pytest

from helpers import random_axes, results_equal
from replica_exchange_wang_landau_b200.engine import Engine, Geometry, RunConfig, System, run_rewl

pytestmark = pytest.mark.gpu

CASES = {  # dimensions, cutoff, windows, walkers, reach, width, couplings, attempts per epoch, epochs
    "two_to_an_sm": ((8, 8, 8), 0.0, 32, 8, 190.0, 0.5, "fp64", 512, 12),
    "two_to_an_sm_width": ((8, 8, 8), 0.0, 32, 8, 190.0, 0.4, "fp64", 301, 12),
    "two_to_an_sm_fp32": ((8, 8, 8), 0.0, 32, 8, 190.0, 0.5, "fp32", 512, 8),
    "two_to_an_sm_bf16": ((8, 8, 8), 0.0, 32, 8, 190.0, 0.5, "bf16", 512, 8),
    "more_than_two": ((8, 8, 8), 0.0, 32, 12, 190.0, 0.5, "fp64", 512, 8),
    "cutoff": ((10, 10, 10), 2.2, 32, 16, 200.0, 0.5, "fp64", 500, 6),
    "sites_4096": ((16, 16, 16), 0.0, 2, 2, 300.0, 1.0, "fp64", 2000, 6),
    "sites_4913": ((17, 17, 17), 0.0, 1, 2, 300.0, 0.75, "fp64", 2000, 6),
}


@pytest.mark.parametrize("name", list(CASES))
def test_pilot_runs(oracle, name):
    dims, cutoff, windows, walkers, reach, width, precision, interval, epochs = CASES[name]
    g = Geometry.simple_cubic(*dims, periodic=True)
    g.axes = random_axes(g.size(), 19)
    s = System(g, 1.0, cutoff)
    half = round(reach / width)
    c = RunConfig(emin=-half * width, emax=half * width, bin_width=width, windows=windows, walkers=walkers, seed=20,
                  overlap=0.75)
    c.exchange_interval_uses_mcs = c.check_interval_uses_mcs = c.max_limit_uses_mcs = False
    c.exchange_interval_attempts, c.wl.check_interval_attempts, c.max_attempts = interval, 4 * interval, epochs * interval
    c.wl.collect_window_statistics = True
    c.coupling_precision, c.recompute_interval_mcs = precision, 0.0
    c.resolve_mcs(s.size())
    with Engine(s, c) as e:
        assert e.sweep == "look-ahead"
    got = run_rewl(s, c)
    assert results_equal(got, oracle.run_rewl(s, c)) == []
    assert len(got.representatives) >= windows * walkers


@pytest.mark.parametrize("epochs_between", [1, 3])
@pytest.mark.parametrize("precision, cutoff", [("fp32", 0.0), ("bf16", 0.0), ("fp32", 1.8)])
def test_representatives_with_a_recompute(oracle, precision, cutoff, epochs_between):
    """An exchanged configuration enters the representatives with the energy it was exchanged with, not with the
    one that the FP64 recompute after the epoch gives it."""
    g = Geometry.simple_cubic(4, 4, 3, periodic=True)
    g.axes = random_axes(48, 19)
    s = System(g, 1.0, cutoff)
    c = RunConfig(emin=-40.0, emax=40.0, bin_width=0.5, windows=4, walkers=3, seed=22, overlap=0.75)
    c.exchange_interval_uses_mcs = c.check_interval_uses_mcs = c.max_limit_uses_mcs = False
    c.exchange_interval_attempts, c.wl.check_interval_attempts, c.max_attempts = 48, 240, 48 * 90
    c.wl.collect_window_statistics = True
    c.coupling_precision, c.recompute_interval_mcs = precision, float(epochs_between)
    c.resolve_mcs(48)
    got = run_rewl(s, c)
    assert got.exchange_accepted > 50 and got.precision_report["recomputes"] >= 29
    assert results_equal(got, oracle.run_rewl(s, c)) == []


@pytest.mark.parametrize("windows, walkers, interval", [(32, 16, 64), (32, 16, 512), (32, 8, 64), (32, 4, 64)])
def test_every_attempt_is_a_sample(windows, walkers, interval):
    """Long runs, epochs launched one by one (more walkers than fit on the GPU at once) and many to a launch: each
    attempt adds one displacement sample, whatever the epochs' ends and the blocks' ends fall on."""
    g = Geometry.simple_cubic(8, 8, 8, periodic=True)
    g.axes = random_axes(512, 19)
    s = System(g)
    c = RunConfig(emin=-190.0, emax=190.0, bin_width=0.5, windows=windows, walkers=walkers, seed=21, overlap=0.75)
    c.exchange_interval_uses_mcs, c.exchange_interval_attempts, c.max_mcs = False, interval, 0.0
    c.wl.collect_window_statistics = True
    c.resolve_mcs(512)
    epochs = 1600 if interval == 64 else 400
    with Engine(s, c) as e:
        for _ in range(4):
            e.run_epochs(epochs // 4)
        samples = sum(int(e.sampling_statistics(w).displacement_samples.sum()) for w in range(windows))
        assert samples == e.totals()["attempted"] == epochs * interval * windows * walkers
