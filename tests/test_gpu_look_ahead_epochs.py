"""Epochs of the look-ahead sweep (csrc/sweep_ahead.cu) that share a launch: what one epoch leaves to the next
and what a failed one leaves behind, bit for bit against the CPU oracle or against epochs launched one by one."""
from __future__ import annotations

import pytest

from helpers import results_equal
from replica_exchange_wang_landau_b200.engine import RunConfig, System, run_rewl
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
