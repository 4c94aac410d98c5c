"""The ring sweep (csrc/sweep.cu) where it runs, with the Nalivaiko mask: walker trajectories and run_rewl
(src/wang_landau.cpp:244-315, src/parallel.cpp:276-747) bit for bit against the oracle, from rows of one
16-site pad to rows of several 512-site chunks, FP64, FP32 and BF16 couplings, bin widths that are and are not
powers of two, pilot statistics, forced acceptance and rejected draws.  (Without the mask dense engines run in
the look-ahead sweep, so every case asserts the sweep.)"""
from __future__ import annotations

import dataclasses

import pytest

from helpers import random_axes, results_equal, snapshots_equal
from test_gpu_rejected_draws import zero_draw_state
from replica_exchange_wang_landau_b200.engine import Engine, Geometry, RunConfig, System, run_rewl

pytestmark = pytest.mark.gpu

# dimensions: couplings rows of 16, 32, 512, 528 and 1104 entries
SIZES = {"n12": (3, 2, 2), "n27": (3, 3, 3), "n512": (8, 8, 8), "n520": (13, 8, 5), "n1089": (11, 11, 9)}


def _system(name):
    g = Geometry.simple_cubic(*SIZES[name], periodic=True)
    g.axes = random_axes(g.size(), 61)
    return System(g, 1.0, 0.0)


def _config(s, steps, precision, seed, **kw):
    """A grid of a few standard deviations of the energy to each side, in steps that are a power of two or not."""
    reach = 2.0 * (1.7 * s.size()) ** 0.5 + 4.0
    width = 2.0 ** -3 if steps == "pow2" else 0.128
    half = round(reach / width)
    c = RunConfig(emin=-half * width, emax=half * width, bin_width=width, windows=2, walkers=2, seed=seed, **kw)
    c.wl.nalivaiko_mod, c.wl.inverse_time_enabled = True, False
    c.coupling_precision = precision
    c.recompute_interval_mcs = 0.0
    return c


@pytest.mark.parametrize("precision", ["fp64", "fp32", "bf16"])
@pytest.mark.parametrize("steps", ["pow2", "other"])
@pytest.mark.parametrize("collect", [False, True])
@pytest.mark.parametrize("name", list(SIZES))
def test_runs(oracle, name, collect, steps, precision):
    s = _system(name)
    mcs = max(4.0, 3000.0 / s.size())
    c = _config(s, steps, precision, 71, max_mcs=mcs, exchange_interval_mcs=mcs / 8, check_interval_mcs=mcs / 4)
    c.wl.collect_window_statistics = collect
    c.wl.flatness, c.wl.minimum_visits = 0.01, 1
    c.resolve_mcs(s.size())
    with Engine(s, c) as e:
        assert e.sweep == "ring"
    got = run_rewl(s, c)
    assert got.accepted > 0
    assert results_equal(got, oracle.run_rewl(s, c)) == []


@pytest.mark.parametrize("name", ["n520", "n1089"])
def test_forced_acceptance(oracle, name):
    s = _system(name)
    c = _config(s, "other", "fp64", 72, max_mcs=8, exchange_interval_mcs=1, check_interval_mcs=2)
    c.force_accept_after_uses_mcs = False
    c.wl.force_accept_after_attempts = 3
    c.resolve_mcs(s.size())
    with Engine(s, c) as e:
        assert e.sweep == "ring"
    got = run_rewl(s, c)
    assert got.forced_accepted > 0
    assert results_equal(got, oracle.run_rewl(s, c)) == []


@pytest.mark.parametrize("collect", [False, True])
@pytest.mark.parametrize("name", ["n27", "n520", "n1089"])
def test_rejected_draws(oracle, name, collect):
    s = _system(name)
    assert ((1 << 64) - s.size()) % s.size() > 0  # a 0 draw is rejected as a site draw
    c = _config(s, "pow2", "fp64", 73)
    c.wl.collect_window_statistics = collect
    c.resolve_mcs(s.size())
    with Engine(s, c) as e:
        assert e.sweep == "ring"
        for w in (0, 3):
            ow = oracle.walker(s, w, c.emin, c.emax, c.bin_width, e.window(w // c.walkers), c.wl, c.seed)
            for rounds, k in enumerate((0, 1, 2, 3, 6, 13, 40)):
                snap = dataclasses.replace(e.snapshot(w), rng_state=zero_draw_state(k, 100 * w + k))
                e.restore(w, snap)
                ow.restore(snap)
                e.run_attempts(w, 150 + 37 * rounds)
                ow.run_attempts(150 + 37 * rounds)
                assert snapshots_equal(e.snapshot(w), ow.snapshot()) == [], f"walker {w}, zero draw {k}"
