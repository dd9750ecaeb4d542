"""Autotuner: candidates that differ, the engine's own default as the one to
beat, strides tuned apart, and choices of older kernels timed again (CPU, with
a stand-in timer)."""
import json

from rtdbstream_gb300 import autotune as AT
from rtdbstream_gb300 import workloads as wl

PTS = wl.gaussian_mixture(30_000, dim=2, k=4, box=20.0, seed=2)


def tuner(tmp_path, table, calls, name="tune.json"):
    def alone(points, dim, W, S, eps, mp, prec, *config):
        calls.append((S, config))
        return table.get(config, 2.0)

    def pool(streams, *config):
        calls.append(("pool", config))
        return table.get(config, 2.0)

    return AT.Autotuner(cache_path=str(tmp_path / name), timer=alone, pool_timer=pool)


def picked(c):
    return c["cell_mult"], c["work_grab"], c["query_lanes"]


def test_candidates_differ_and_start_with_the_engine_default():
    # a warp takes max(1, grab / 16) blocks of positions
    assert len({(k, max(1, grab >> 4), lanes) for k, grab, lanes in AT.CANDIDATES}) == len(AT.CANDIDATES)
    assert AT.CANDIDATES[0] == (1, 0, 0)
    assert {(k, max(1, grab >> 4)) for k, grab, _ in AT.CANDIDATES} == {(1, 1), (1, 2), (2, 1), (2, 2)}


def test_engine_default_is_kept_within_the_margin(tmp_path):
    t = tuner(tmp_path, {(1, 0, 0): 1.0, (1, 8, 16): 0.98, (1, 8, 32): 0.99, (2, 8, 32): 0.975}, [])
    assert picked(t.choose(PTS, 2, 10_000, 500, 0.5, 5)) == (1, 0, 0)
    assert picked(t.choose_batched([(PTS, 2, 10_000, 500, 0.5, 5, "fp64")])[0]) == (1, 0, 0)


def test_strides_are_tuned_apart(tmp_path):
    calls = []
    t = tuner(tmp_path, {(1, 8, 32): 1.0}, calls)
    t.choose(PTS, 2, 10_000, 100, 0.5, 5)
    t.choose(PTS, 2, 10_000, 5_000, 0.5, 5)
    assert {s for s, _ in calls} == {100, 5_000} and t.tuned == 2
    calls.clear()
    t.choose(PTS, 2, 10_000, 110, 0.5, 5)  # of the first one's bucket
    assert not calls


def test_choices_of_older_kernels_are_timed_again(tmp_path):
    calls = []
    t = tuner(tmp_path, {(2, 8, 32): 1.0}, calls)
    stream = (PTS, 2, 10_000, 500, 0.5, 5, "fp64")
    t.choose(*stream)
    t.choose_batched([stream])
    saved = json.loads((tmp_path / "tune.json").read_text())
    assert len(saved) == 2
    for entry in saved.values():
        entry.pop("kernels")
    (tmp_path / "old.json").write_text(json.dumps(saved))
    calls.clear()
    old = tuner(tmp_path, {(1, 8, 32): 1.0}, calls, "old.json")
    assert picked(old.choose(*stream)) == (1, 8, 32) and len(calls) == len(AT.CANDIDATES)
    assert picked(old.choose_batched([stream])[0]) == (1, 8, 32) and len(calls) == 2 * len(AT.CANDIDATES)
