"""Which sweep runs which engine, and its trajectories bit for bit against the CPU oracle on both sides of
every rule (results never depend on the route)."""
from __future__ import annotations

import pytest

from helpers import random_axes, results_equal
from replica_exchange_wang_landau_b200.engine import Engine, Geometry, InvalidArgument, RunConfig, System, run_rewl

pytestmark = pytest.mark.gpu


def _lattice(dims, seed, cutoff=0.0):
    g = Geometry.simple_cubic(*dims, periodic=True)
    g.axes = random_axes(g.size(), seed)
    return System(g, 1.0, cutoff)


def _check(oracle, s, c, sweep):
    c.resolve_mcs(s.size())
    with Engine(s, c) as e:
        assert e.sweep == sweep
    got = run_rewl(s, c)
    assert got.attempted > 0
    assert results_equal(got, oracle.run_rewl(s, c)) == []


# A window's bins in the look-ahead sweep take 16 bytes each beside 57 KB, in the ring sweep 17 beside four rows.
@pytest.mark.parametrize("precision", ["fp64", "fp32", "bf16"])
@pytest.mark.parametrize("bins, sweep", [(9000, "look-ahead"), (11500, "ring")])
def test_wide_windows(oracle, bins, sweep, precision):
    s = _lattice((4, 4, 4), 3)
    for width in (2.0 ** -7, 0.009):
        c = RunConfig(emin=-(bins // 2) * width, emax=(bins // 2) * width, bin_width=width, windows=1, walkers=2,
                      seed=11, max_mcs=60, exchange_interval_mcs=2, check_interval_mcs=6)
        c.coupling_precision = precision
        _check(oracle, s, c, sweep)


@pytest.mark.parametrize("precision", ["fp64", "bf16"])
def test_staging_depths_are_those_that_fit(oracle, precision):
    """Six block records fit beside the walker wherever the look-ahead sweep has a staging depth; an engine whose
    window is too wide for that sweep has none."""
    s = _lattice((9, 10, 11), 4)
    c = RunConfig(emin=-400, emax=400, bin_width=1.0, windows=2, walkers=2, seed=12, max_mcs=6,
                  exchange_interval_mcs=1, check_interval_mcs=2)
    c.coupling_precision = precision
    c.resolve_mcs(s.size())
    with Engine(s, c) as e:
        assert e.sweep == "look-ahead"
        e.set_staging_ring(32)
        e.run()
        got = e.result()
    assert results_equal(got, oracle.run_rewl(s, c)) == []
    s = _lattice((4, 4, 4), 3)
    c = RunConfig(emin=-5750 * 2.0 ** -7, emax=5750 * 2.0 ** -7, bin_width=2.0 ** -7, windows=1, walkers=2, seed=11)
    c.coupling_precision = precision
    c.resolve_mcs(s.size())
    with Engine(s, c) as e:
        assert e.sweep == "ring"
        for entries in (16, 32):
            with pytest.raises(InvalidArgument):
                e.set_staging_ring(entries)


AUTOTUNE = {  # (cutoff, pilot statistics, Nalivaiko mask, sweep, candidates, passes)
    "dense": (0.0, False, False, "look-ahead", 2, 6),  # the two staging depths
    "pilot": (0.0, True, False, "look-ahead", 1, 6),
    "cutoff": (1.8, False, False, "look-ahead", 1, 6),
    "mask": (0.0, False, True, "ring", 5, 2),  # epochs per graph replay
    "cutoff_mask": (1.8, False, True, "generic", 20, 2),  # ... and walkers per CTA
}


@pytest.mark.parametrize("name", list(AUTOTUNE))
def test_autotune_varies_what_the_launches_depend_on(name):
    cutoff, pilot, mask, sweep, candidates, passes = AUTOTUNE[name]
    s = _lattice((4, 4, 4), 3, cutoff)
    c = RunConfig(emin=-60, emax=60, bin_width=0.5, windows=2, walkers=2, overlap=0.5, seed=9)
    c.wl.collect_window_statistics, c.wl.nalivaiko_mod = pilot, mask
    c.wl.inverse_time_enabled = not mask
    c.exchange_interval_mcs, c.max_mcs = 2.0, 1e6
    c.resolve_mcs(s.size())
    with Engine(s, c) as e:
        assert e.sweep == sweep
        e.set_launch(0, 10)
        r = e.autotune(4)
        assert r["trials"] == candidates * passes and r["ms_per_epoch"] > 0
        assert (r["epochs_per_graph"] == 10) == (passes == 6)
