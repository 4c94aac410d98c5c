"""The split sweep (csrc/sweep_split.cu): the rules that choose it, and runs on both sides of its chunks of 64
sites bit for bit against the CPU oracle -- exchanges, the 1/t stage, forced acceptance, rejected draws, the FP64
recompute, both staging depths, three precisions, widths that are and are not powers of two."""
from __future__ import annotations

import dataclasses

import pytest

from helpers import random_axes, results_equal, snapshots_equal
from test_gpu_rejected_draws import zero_draw_state
from replica_exchange_wang_landau_b200.engine import (DeviceError, Engine, Geometry, RunConfig, System, run_rewl)
from replica_exchange_wang_landau_b200.geometry import simple_cubic_random

pytestmark = pytest.mark.gpu

SITES = (1, 12, 16, 17, 48, 64, 65, 128, 129, 200, 256, 257, 512)


def _row(n):
    return System(simple_cubic_random(n, 1, 1, seed=n, periodic=False))


def _config(windows, walkers, interval, attempts, width=0.25, precision="fp64", reach=80.0, **wl):
    half = round(reach / width)
    c = RunConfig(emin=-half * width, emax=half * width, bin_width=width, windows=windows, walkers=walkers, seed=17)
    c.exchange_interval_uses_mcs = c.check_interval_uses_mcs = c.max_limit_uses_mcs = False
    c.exchange_interval_attempts, c.wl.check_interval_attempts, c.max_attempts = interval, 5 * interval, attempts
    c.coupling_precision, c.recompute_interval_mcs = precision, 0.0
    for k, v in wl.items():
        setattr(c.wl, k, v)
    return c


def _run(oracle, s, c, sweep="split", staging=0):
    c.resolve_mcs(s.size())
    with Engine(s, c) as e:
        assert e.sweep == sweep
        if staging:
            e.set_staging_ring(staging)
        e.run()
        got = e.result()
    assert results_equal(got, oracle.run_rewl(s, c)) == []
    return got


@pytest.mark.parametrize("precision", ["fp64", "fp32", "bf16"])
@pytest.mark.parametrize("n", SITES)
def test_sites(oracle, n, precision):
    """More walkers than SMs and epochs of at most 32 attempts."""
    for width, staging in ((0.25, 16), (0.3, 32)):
        _run(oracle, _row(n), _config(2, 75, 29, 2900, width, precision), staging=staging)


@pytest.mark.parametrize("dims, windows, walkers", [((3, 3, 3), 4, 112), ((4, 4, 4), 4, 112), ((6, 6, 6), 4, 75)])
def test_more_walkers_than_fit(oracle, dims, windows, walkers):
    g = Geometry.simple_cubic(*dims, periodic=True)
    g.axes = random_axes(g.size(), 3)
    got = _run(oracle, System(g), _config(windows, walkers, 65, 650, 0.5, reach=60.0))
    assert got.exchange_accepted > 0


def test_inverse_time_stage(oracle):
    g = Geometry.simple_cubic(3, 3, 2, periodic=True)
    g.axes = random_axes(18, 3)
    for width in (2.0, 2.1):
        got = _run(oracle, System(g), _config(2, 75, 31, 31000, width, reach=32.0, minimum_visits=1, final_factor=1e-3))
        assert all(w["factor"] < 0.01 for w in got.walker_statistics)


def test_forced_acceptance(oracle):
    g = Geometry.simple_cubic(3, 2, 2, periodic=False)
    c = _config(2, 75, 30, 900, reach=30.0, force_accept_after_attempts=3)
    c.force_accept_after_uses_mcs = False
    assert _run(oracle, System(g), c).forced_accepted > 0


@pytest.mark.parametrize("width", [0.25, 0.3])
def test_rejected_draws(oracle, width):
    g = Geometry.simple_cubic(3, 3, 3, periodic=True)
    g.axes = random_axes(27, 31)
    s = System(g)
    c = _config(2, 75, 32, 0, width, reach=60.0)
    c.resolve_mcs(27)
    with Engine(s, c) as e:
        assert e.sweep == "split"
        for w in (0, 149):
            ow = oracle.walker(s, w, c.emin, c.emax, c.bin_width, e.window(w // c.walkers), c.wl, c.seed)
            for rounds, k in enumerate((0, 1, 2, 3, 6, 13, 40)):
                snap = dataclasses.replace(e.snapshot(w), rng_state=zero_draw_state(k, 100 * w + k))
                e.restore(w, snap)
                ow.restore(snap)
                e.run_attempts(w, 150 + 37 * rounds)
                ow.run_attempts(150 + 37 * rounds)
                assert snapshots_equal(e.snapshot(w), ow.snapshot()) == [], f"walker {w}, zero draw {k}"


@pytest.mark.parametrize("precision, interval, sweep", [("fp32", 8, "split"), ("fp32", 32, "split"),
                                                        ("fp32", 33, "look-ahead"), ("bf16", 64, "split"),
                                                        ("bf16", 65, "look-ahead")])
def test_epochs_with_a_recompute_each(oracle, precision, interval, sweep):
    g = Geometry.simple_cubic(3, 3, 3, periodic=True)
    g.axes = random_axes(27, 31)
    c = _config(2, 2, interval, 40 * interval, precision=precision, reach=60.0)
    c.recompute_interval_mcs, c.recompute_interval_attempts = interval / 27.0, interval
    got = _run(oracle, System(g), c, sweep)
    assert got.precision_report["recomputes"] == 39  # after every epoch but the last


@pytest.mark.parametrize("walkers, interval, sweep", [(74, 32, "look-ahead"), (75, 32, "split"), (75, 33, "look-ahead"),
                                                      (185, 64, "look-ahead"), (186, 64, "split"),
                                                      (222, 65, "look-ahead"), (223, 65, "split")])
def test_rules(oracle, walkers, interval, sweep):
    """64 sites, two windows; of 148 SMs, on each of which three walkers of the look-ahead sweep fit."""
    g = Geometry.simple_cubic(4, 4, 4, periodic=True)
    g.axes = random_axes(64, 3)
    _run(oracle, System(g), _config(2, walkers, interval, 50 * interval, 0.5, reach=60.0), sweep)


def test_wait_runs_out():
    g = Geometry.simple_cubic(3, 3, 3, periodic=True)
    c = _config(2, 75, 30, 0, reach=60.0)
    c.resolve_mcs(27)
    with Engine(System(g), c) as e:
        assert e.sweep == "split"
        before = [e.snapshot(w) for w in range(e.walkers)]
        e.inject_wait_timeout()
        with pytest.raises(DeviceError) as err:
            e.run_epochs(3)
        assert err.value.status == "WLG_ERR_TIMEOUT"
        assert all(snapshots_equal(e.snapshot(w), before[w]) == [] for w in range(e.walkers))
