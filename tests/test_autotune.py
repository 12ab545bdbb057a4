"""Host side of the autotuner (master_b200/autotune.py): its JSON cache and
how a cached choice is found for a workload, without a GPU."""
from __future__ import annotations

import json

import pytest

from master_b200 import autotune


def test_cache_path_honours_the_environment(tmp_path, monkeypatch):
    monkeypatch.setenv("DSMC_TUNE_CACHE", str(tmp_path / "t.json"))
    assert autotune.cache_path() == tmp_path / "t.json"
    monkeypatch.delenv("DSMC_TUNE_CACHE")
    monkeypatch.setenv("XDG_CACHE_HOME", str(tmp_path / "xdg"))
    assert autotune.cache_path() == tmp_path / "xdg" / "dsmc_b200" / "tuning.json"


def test_cache_round_trip_and_unreadable_files(tmp_path, monkeypatch):
    p = tmp_path / "sub" / "tuning.json"
    monkeypatch.setenv("DSMC_TUNE_CACHE", str(p))
    assert autotune.load_cache() == {}          # no file yet
    entries = {"k": {"choice": {"blocks_per_sm": [0, 4, 0, 5, 0], "ring": 0, "collide_claim": 2}}}
    autotune.save_cache(entries)
    assert autotune.load_cache() == entries
    assert not p.with_suffix(".tmp").exists()   # written through a temporary file, then renamed
    p.write_text("{not json")
    assert autotune.load_cache() == {}


def test_signature_key_ignores_field_order():
    a = {"gpu": "NVIDIA B200", "sms": 148, "cells": 1 << 21, "particles": 1 << 25, "min_ring": 96, "pipelined": 1}
    b = dict(reversed(list(a.items())))
    assert autotune._key(a) == autotune._key(b)
    assert autotune._key(a) != autotune._key({**a, "sms": 132})


@pytest.mark.parametrize("x,want", [(0, 0), (-3, 0), (1, 1), (3, 4), (5, 4), (6, 8), (1000, 1024), (31_478_288, 1 << 25)])
def test_workload_sizes_round_to_powers_of_two(x, want):
    assert autotune._pow2(x) == want


def test_apply_cached_sets_the_stored_choice(tmp_path, monkeypatch):
    monkeypatch.setenv("DSMC_TUNE_CACHE", str(tmp_path / "tuning.json"))
    sig = {"gpu": "NVIDIA B200", "sms": 148, "cells": 4096, "particles": 1 << 19, "min_ring": 64, "pipelined": 1}
    choice = {"blocks_per_sm": [2, 4, 0, 5, 0], "ring": 128, "collide_claim": 1}
    autotune.save_cache({autotune._key(sig): {"choice": choice, "default_ms": {}, "chosen_ms": {}}})
    calls = []
    monkeypatch.setattr(autotune, "set_tuning", lambda ctx, bps, ring, claim: calls.append((ctx, bps, ring, claim)))
    monkeypatch.setattr(autotune, "signature", lambda ctx: dict(sig))
    ctx = object()
    entry = autotune.apply_cached(ctx)
    assert entry["choice"] == choice
    assert calls == [(ctx, choice["blocks_per_sm"], 128, 1)]
    # another workload: nothing cached, nothing set
    monkeypatch.setattr(autotune, "signature", lambda ctx: {**sig, "cells": 8192})
    assert autotune.apply_cached(ctx) is None
    assert len(calls) == 1
    assert json.loads((tmp_path / "tuning.json").read_text())  # the cache itself untouched


class FakeContext:
    """A context whose kernels take the times `ms` gives for a launch shape."""

    def __init__(self, ms, limits=(2, 2, 4, 3, 2), ring=128, launches=lambda bps: 4):
        self.ms, self.limits, self.ring, self.launches = ms, limits, ring, launches
        self.set = ((0,) * 5, 0, 0)

    def pass_info(self):
        return {"pipelined": 1}

    def pass_launches(self):
        return self.launches(self.set[0]), 1

    def step(self, n):
        pass

    def set_timing(self, on):
        pass

    def pass_times(self):
        return {**dict(zip(autotune.KERNELS, self.ms(*self.set))), "passes": 1}


def tuned(ctx, monkeypatch):
    from master_b200 import capi

    def set_tuning(ctx, bps=(0,) * 5, ring=0, claim=0):
        ctx.set = (tuple(bps), ring, claim)

    def get(ctx):
        lim = capi.Tuning()
        for k, b in enumerate(ctx.limits):
            lim.blocks_per_sm[k] = b
        lim.ring = max(ctx.ring, ctx.set[1])
        return capi.Tuning(), lim

    monkeypatch.setattr(autotune, "set_tuning", set_tuning)
    monkeypatch.setattr(autotune, "get", get)
    monkeypatch.setattr(autotune, "signature", lambda ctx: {})
    return autotune.tune(ctx, steps=1, repeats=1, store=False)


def test_tuner_weighs_place_movers_with_the_flights_it_hands_on(monkeypatch):
    """With fewer than three blocks per SM place_movers lists its wall flights and
    its own time drops by less than place_walls' rises: the default stays for
    it, and the other kernels keep their better shapes."""
    def ms(bps, ring, claim):
        place = bps[2] or 4
        return (0.5 if bps[0] == 1 and claim == 2 else 1.0, 0.6 if bps[1] == 1 else 1.0,
                1.0 if place >= 3 else 0.6, 0.0 if place >= 3 else 0.9)
    rep = tuned(FakeContext(ms, launches=lambda bps: 3 if (bps[2] or 4) >= 3 else 4), monkeypatch)
    assert rep["choice"] == {"blocks_per_sm": [1, 1, 0, 0, 0], "ring": 0, "collide_claim": 2}


def test_tuner_leaves_a_kernel_alone_that_does_not_run(monkeypatch):
    """place_walls not launched: what its interval reads is noise, not a choice."""
    def ms(bps, ring, claim):
        return 1.0, 1.0, 1.0, 1e-6 if bps[3] == 0 else 5e-7
    rep = tuned(FakeContext(ms, launches=lambda bps: 3), monkeypatch)
    assert rep["choice"]["blocks_per_sm"][3] == 0


def test_tuner_times_place_walls_as_it_runs_with_the_chosen_place_movers(monkeypatch):
    """The chosen place_movers grid lists its flights: place_walls' blocks are
    compared with that grid set, not with the default's."""
    def ms(bps, ring, claim):
        if (bps[2] or 4) >= 3:
            return 1.0, 1.0, 2.0, 0.0
        return 1.0, 1.0, 0.6, 0.5 if bps[3] == 2 else 0.8
    rep = tuned(FakeContext(ms, launches=lambda bps: 3 if (bps[2] or 4) >= 3 else 4), monkeypatch)
    assert rep["choice"]["blocks_per_sm"] == [0, 0, 1, 2, 0]


def test_tuner_tries_the_staging_sizes_there_are(monkeypatch):
    rep = tuned(FakeContext(lambda bps, ring, claim: (1.0, 1.0 - ring * 1e-4, 1.0, 1.0), ring=160), monkeypatch)
    assert rep["choice"]["ring"] == 224
    assert min(autotune.RINGS) == 128
