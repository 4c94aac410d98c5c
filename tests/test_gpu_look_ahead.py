"""The look-ahead sweep at the edges of its blocks, tiles and rules, bit for bit against the CPU oracle:
the trajectories are exact by construction, so every comparison is one of equality."""
from __future__ import annotations

import pytest

from helpers import results_equal, snapshots_equal
from replica_exchange_wang_landau_b200.engine import Batch, DeviceError, Engine, RunConfig, System, run_rewl
from replica_exchange_wang_landau_b200.geometry import simple_cubic_random

pytestmark = pytest.mark.gpu

# A block holds 30 draws and hands two on; a warp takes 32 pairs; the field warps take tiles of 64 sites.
SITES = (1, 2, 15, 16, 17, 31, 32, 33, 63, 64, 65, 127, 129, 257)
INTERVALS = (1, 29, 30, 31, 32, 61, 600)


def _config(width, interval, attempts, **kw):
    c = RunConfig(emin=-400 * width, emax=400 * width, bin_width=width, **kw)
    c.exchange_interval_uses_mcs = c.check_interval_uses_mcs = c.max_limit_uses_mcs = False
    c.exchange_interval_attempts = interval
    c.wl.check_interval_attempts = 7 * interval
    c.max_attempts = attempts
    c.wl.final_factor = 1e-4
    return c


def _row(n, seed, cutoff=0.0):
    return System(simple_cubic_random(n, 1, 1, seed=seed, periodic=False), 1.0, cutoff)


@pytest.mark.parametrize("n", SITES)
def test_sites(oracle, n):
    """Widths that are powers of two and ones that are not, two windows with exchanges."""
    for width in (0.25, 0.3):
        c = _config(width, 47, 4000, windows=2, walkers=2, seed=100 + n, overlap=0.75)
        c.resolve_mcs(n)
        s = _row(n, n)
        assert results_equal(run_rewl(s, c), oracle.run_rewl(s, c)) == []


@pytest.mark.parametrize("precision", ["fp64", "fp32", "bf16"])
@pytest.mark.parametrize("n", SITES)
def test_epochs_to_a_launch(n, precision):
    """Epochs many to a launch and epochs as launches of their own leave the same walkers."""
    c = _config(0.25, 47, 10_000_000, windows=2, walkers=2, seed=200 + n, overlap=0.75)
    c.coupling_precision = precision
    c.recompute_interval_mcs = 0.0
    c.resolve_mcs(n)
    with Engine(_row(n, n), c) as a, Engine(_row(n, n), c) as b:
        a.run_epochs(25)
        b.time_epochs(25)
        for w in range(a.walkers):
            assert snapshots_equal(a.snapshot(w), b.snapshot(w)) == []
        assert a.totals()["attempted"] > 0


@pytest.mark.parametrize("collect", [False, True])
@pytest.mark.parametrize("interval", INTERVALS)
def test_exchange_intervals(oracle, interval, collect):
    """Batches that end before, on and after the end of a block, with exchanges between windows."""
    s = System(simple_cubic_random(3, 3, 2, seed=5, periodic=True))
    for width in (0.25, 0.3):
        c = _config(width, interval, 3000, windows=3, walkers=2, seed=7, overlap=0.75)
        c.emin, c.emax = -160 * width, 160 * width
        c.wl.collect_window_statistics = collect
        c.resolve_mcs(s.size())
        assert results_equal(run_rewl(s, c), oracle.run_rewl(s, c)) == []


@pytest.mark.parametrize("force", [1, 3, 40])
def test_forced_acceptance(oracle, force):
    s = System(simple_cubic_random(3, 2, 2, seed=6, periodic=False))
    c = _config(0.25, 30, 3000, windows=2, walkers=2, seed=8, overlap=0.75)
    c.emin, c.emax = -30.0, 30.0
    c.force_accept_after_uses_mcs = False
    c.wl.force_accept_after_attempts = force
    c.resolve_mcs(s.size())
    got = run_rewl(s, c)
    assert results_equal(got, oracle.run_rewl(s, c)) == []
    assert got.forced_accepted > 0 or force > 3


@pytest.mark.parametrize("n", [2047, 2048, 2049])
def test_cutoff_full_rows(oracle, n):
    """Cutoff systems on both sides of the size up to which they have full rows."""
    s = _row(n, 3, 1.8)
    c = _config(4.0, 300, 1500, windows=2, walkers=2, seed=9, overlap=0.75)
    c.emin, c.emax = -5000.0, 5000.0
    c.resolve_mcs(n)
    assert results_equal(run_rewl(s, c), oracle.run_rewl(s, c)) == []


def test_batch_after_epochs():
    """An engine that has run a graph's worth of epochs enters a batch as it is; one that has not runs one first."""
    c = _config(0.25, 47, 10_000_000, windows=2, walkers=2, seed=11, overlap=0.75)
    c.resolve_mcs(33)
    for before, extra in ((8, 0), (7, 1)):
        with Engine(_row(33, 4), c) as a, Engine(_row(33, 4), c) as b:
            a.set_launch(0, 8)
            a.run_epochs(before)
            with Batch([a]) as batch:
                assert a.totals()["epochs"] == before + extra
                batch.run_epochs(8)
            b.run_epochs(before + extra + 8)
            assert a.totals()["epochs"] == b.totals()["epochs"]
            for w in range(a.walkers):
                assert snapshots_equal(a.snapshot(w), b.snapshot(w)) == []


@pytest.mark.parametrize("n", [1, 16, 17, 32])
@pytest.mark.parametrize("interval", [31, 32, 33, 200000])
def test_single_window_rule(oracle, n, interval):
    """Single-window engines on both sides of the interval from which the look-ahead sweep takes their epochs,
    and beyond the longest epoch that shares a launch."""
    for width in (0.25, 0.3):
        c = _config(width, interval, 300000 if interval > 100 else 3000, windows=1, walkers=2, seed=n)
        c.emin, c.emax = -160 * width, 160 * width
        c.wl.check_interval_attempts = 10 * interval
        c.resolve_mcs(n)
        s = _row(n, n)
        with Engine(s, c) as e:
            assert e.window_sweep
        assert results_equal(run_rewl(s, c), oracle.run_rewl(s, c)) == []


@pytest.mark.parametrize("interval", [8, 80])
def test_single_window_wait_runs_out(interval):
    c = _config(0.25, interval, 3000, windows=1, walkers=2, seed=3)
    c.resolve_mcs(8)
    with Engine(_row(8, 2), c) as e:
        before = [e.snapshot(w) for w in range(e.walkers)]
        e.inject_wait_timeout()
        with pytest.raises(DeviceError) as err:
            e.run()
        assert err.value.status == "WLG_ERR_TIMEOUT"
        assert all(snapshots_equal(e.snapshot(w), before[w]) == [] for w in range(e.walkers))
