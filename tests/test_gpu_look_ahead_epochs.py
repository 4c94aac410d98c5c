"""Epochs of the look-ahead sweep (csrc/sweep_ahead.cu) that share a launch: what one epoch leaves to the next
and what a failed one leaves behind, bit for bit against the CPU oracle or against epochs launched one by one."""
from __future__ import annotations

import dataclasses

import numpy as np
import pytest

from helpers import results_equal, same_double, snapshots_equal
from replica_exchange_wang_landau_b200.engine import (DeviceError, Engine, EscapedError, RunConfig, System, WlgError,
                                                      run_rewl)
from replica_exchange_wang_landau_b200.geometry import simple_cubic_random

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("inverse_time", [True, False])
@pytest.mark.parametrize("interval", [1, 2, 3, 5])
def test_exchanges_into_unvisited_bins(oracle, interval, inverse_time):
    """Bins so fine that an exchange nearly always brings one not visited before, and epochs so short that
    their first attempts fall on every draw of a block, its last one included."""
    s = System(simple_cubic_random(3, 3, 2, seed=5, periodic=True))
    for width in (2.0 ** -8, 0.003):
        c = RunConfig(emin=-36.0, emax=36.0, bin_width=width, windows=12, walkers=6, seed=13,
                      overlap=0.75)
        c.exchange_interval_uses_mcs = c.check_interval_uses_mcs = c.max_limit_uses_mcs = False
        c.exchange_interval_attempts = interval
        c.wl.check_interval_attempts = 50 * interval
        c.wl.inverse_time_enabled = inverse_time
        c.max_attempts = 4500
        c.resolve_mcs(s.size())
        got = run_rewl(s, c)
        assert got.exchange_accepted > 100
        assert results_equal(got, oracle.run_rewl(s, c)) == []


def _failing_config(collect, width=0.25):
    c = RunConfig(emin=-160 * width, emax=160 * width, bin_width=width, windows=3, walkers=2, seed=7, overlap=0.75)
    c.exchange_interval_uses_mcs = c.check_interval_uses_mcs = c.max_limit_uses_mcs = False
    c.exchange_interval_attempts = 47
    c.wl.check_interval_attempts = 3 * 47
    c.wl.flatness, c.wl.minimum_visits = 0.01, 1
    c.wl.collect_window_statistics = collect
    c.max_attempts = 1_000_000
    return c


def _same_state(a, b, collect):
    assert a.totals() == b.totals()
    for w in range(a.walkers):
        assert snapshots_equal(a.snapshot(w), b.snapshot(w)) == [], f"walker {w}"
    if collect:
        for window in range(3):
            sa, sb = a.sampling_statistics(window), b.sampling_statistics(window)
            assert same_double(sa.squared_energy_displacement, sb.squared_energy_displacement)
            assert np.array_equal(sa.displacement_samples, sb.displacement_samples)
            assert sa.round_trips == sb.round_trips


@pytest.mark.parametrize("collect", [False, True])
@pytest.mark.parametrize("walker, blocks", [(0, 0), (3, 0), (0, 7), (2, 13), (5, 31)])
def test_a_wait_that_runs_out_within_a_launch(walker, blocks, collect):
    """The epoch in which it happens ends the run: the others have made it, the failed walker is where it was
    before it, as when that epoch is launched by itself."""
    s = System(simple_cubic_random(3, 3, 2, seed=5, periodic=True))
    c = _failing_config(collect)
    c.resolve_mcs(s.size())
    with Engine(s, c) as a, Engine(s, c) as b:
        a.run_epochs(20)
        b.run_epochs(20)
        a.inject_wait_timeout(walker, blocks)
        with pytest.raises(DeviceError) as err:
            a.run_epochs(60)
        assert err.value.status == "WLG_ERR_TIMEOUT"
        made = a.totals()["epochs"] - 20
        assert made == 0 if blocks == 0 else 0 < made < 60
        b.run_epochs(made)
        b.inject_wait_timeout(walker, 0)
        with pytest.raises(DeviceError):
            b.time_epochs(1)
        _same_state(a, b, collect)


@pytest.mark.parametrize("collect", [False, True])
def test_an_escaped_walker_leaves_the_others_whole(collect):
    """A walker restored with an energy outside its window ends the run with the launch's first epoch."""
    s = System(simple_cubic_random(3, 3, 2, seed=5, periodic=True))
    c = _failing_config(collect)
    c.resolve_mcs(s.size())
    with Engine(s, c) as a, Engine(s, c) as b:
        for e in (a, b):
            e.run_epochs(20)
            with pytest.raises(WlgError):  # the state is replaced before the energy is found wrong
                e.restore(3, dataclasses.replace(e.snapshot(3), energy=1e6))
        with pytest.raises(EscapedError):
            a.run_epochs(60)
        before = [b.snapshot(w) for w in range(b.walkers)]
        for w in (0, 1, 2, 4, 5):
            b.run_attempts(w, c.exchange_interval_attempts)
        assert a.totals()["epochs"] == 20
        for w in range(a.walkers):
            got, want = a.snapshot(w), b.snapshot(w)
            if w == 3:
                assert snapshots_equal(got, before[w]) == []
            else:  # (run_attempts makes no check: the histogram and the stage are the epoch's)
                for k in ("spins", "active"):
                    assert np.array_equal(getattr(got, k), getattr(want, k))
                for k in ("fields", "log_g"):
                    assert same_double(getattr(got, k), getattr(want, k))
                assert (got.energy, got.attempted, got.accepted, got.rng_state) == \
                    (want.energy, want.attempted, want.accepted, want.rng_state)
