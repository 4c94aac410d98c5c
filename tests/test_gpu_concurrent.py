"""Engines driven from several host threads at once, each from its own: launches of several epochs wait for the
other walkers of their own engine, so they have to start with all of them resident, whatever else the GPU
runs.  Neither engine's walkers fit beside the other's.  Results are those of each engine by itself."""
from __future__ import annotations

import threading

import pytest

from helpers import random_axes, snapshots_equal
from replica_exchange_wang_landau_b200.engine import Batch, Engine, Geometry, RunConfig, System

pytestmark = pytest.mark.gpu


def _system():
    g = Geometry.simple_cubic(8, 8, 8, periodic=True)
    g.axes = random_axes(512, 3)
    return System(g, 1.0, 0.0)


def _engine(s, seed, windows=16, walkers=8, interval=512):
    c = RunConfig(emin=-190, emax=190, bin_width=0.5, windows=windows, walkers=walkers, seed=seed)
    c.exchange_interval_uses_mcs, c.exchange_interval_attempts, c.max_mcs = False, interval, 0.0
    c.resolve_mcs(s.size())
    return Engine(s, c)


def _together(*work):
    errors = []

    def run(f):
        try:
            f()
        except Exception as e:  # noqa: BLE001 (reported below)
            errors.append(e)

    threads = [threading.Thread(target=run, args=(f,)) for f in work]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert errors == []


def _states(e):
    return [e.snapshot(w) for w in range(e.walkers)]


def _same(a, b):
    assert all(snapshots_equal(x, y) == [] for x, y in zip(a, b)) and len(a) == len(b)


def test_two_engines_in_two_threads():
    s = _system()
    want = []
    for seed in (1, 2):
        with _engine(s, seed) as e:
            e.run_epochs(400)
            want.append(_states(e))
    with _engine(s, 1) as a, _engine(s, 2) as b:
        _together(lambda: [a.run_epochs(40) for _ in range(10)], lambda: [b.run_epochs(40) for _ in range(10)])
        _same(_states(a), want[0])
        _same(_states(b), want[1])


def test_an_engine_beside_a_batch():
    s = _system()
    with _engine(s, 3) as e:
        e.run_epochs(400)
        want = _states(e)
    engines = [_engine(s, 100 + k, windows=1, walkers=2, interval=16384) for k in range(30)]
    try:
        for e in engines:
            e.set_launch(0, 8)
        with _engine(s, 3) as a, Batch(engines) as batch:
            _together(lambda: [a.run_epochs(40) for _ in range(10)], lambda: batch.run_epochs(40))
            _same(_states(a), want)
        with _engine(s, 100, windows=1, walkers=2, interval=16384) as b:
            b.run_epochs(engines[0].totals()["epochs"])
            _same(_states(engines[0]), _states(b))
    finally:
        for e in engines:
            e.close()
