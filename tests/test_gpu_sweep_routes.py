"""Which sweep runs which engine, and its trajectories bit for bit against the CPU oracle on both sides of
every rule (results never depend on the route)."""
from __future__ import annotations

import pytest

from helpers import random_axes, results_equal
from replica_exchange_wang_landau_b200.engine import Engine, Geometry, RunConfig, System, run_rewl

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
