"""The launch-schedule autotuner's host logic (CPU: a fake timer stands in
for the CUDA-event timing; set_schedule only records host state)."""
import json

import pytest

from openifs_b200 import autotune, cloudsc


@pytest.fixture
def restore_schedule():
    saved = {p: cloudsc.get_schedule(p) for p in (cloudsc.FP64, cloudsc.MIXED)}
    yield
    for p, s in saved.items():
        cloudsc.set_schedule(p, *s)


def test_candidates_are_valid(restore_schedule):
    for prec in (cloudsc.FP64, cloudsc.MIXED):
        cands = autotune.candidates(prec)
        assert len(cands) == len(set(cands)) >= cloudsc.num_variants()
        for v, t, c in cands:
            info = cloudsc.variant_info(prec, v)
            assert t % 32 == 0 and 32 <= t <= info["max_threads"]
            assert c in (0, info["min_ctas"])
            cloudsc.set_schedule(prec, v, t, c)
            assert cloudsc.get_schedule(prec) == (v, t, c)


def test_schedule_limits(restore_schedule):
    n = cloudsc.num_variants()
    info = [cloudsc.variant_info(cloudsc.FP64, v) for v in range(n)]
    big = max(range(n), key=lambda v: info[v]["max_threads"])
    with pytest.raises(cloudsc.CloudscError):
        cloudsc.set_schedule(cloudsc.FP64, big, info[big]["max_threads"] + 32, 0)
    with pytest.raises(cloudsc.CloudscError):
        cloudsc.set_schedule(cloudsc.FP64, n, 128, 0)
    with pytest.raises(cloudsc.CloudscError):
        cloudsc.set_schedule(cloudsc.FP64, 0, 100, 0)
    # set_launch: the one-CTA-per-SM variant with the most registers that fits
    cloudsc.set_launch(cloudsc.FP64, 128, 0)
    v, t, c = cloudsc.get_schedule(cloudsc.FP64)
    fits = [u for u in range(n) if info[u]["min_ctas"] == 1 and info[u]["max_threads"] >= 128]
    assert t == 128 and info[v]["max_threads"] == min(info[u]["max_threads"] for u in fits)


def test_setting_what_is_reported_changes_nothing(restore_schedule):
    """A set schedule can be taken back: the default, each call by its number of
    columns, reads as 0 threads and is restored by setting what was read."""
    for prec in (cloudsc.FP64, cloudsc.MIXED, cloudsc.PHYS32):
        default = cloudsc.get_schedule(prec)
        assert default[1:] == (0, 0)
        cloudsc.set_schedule(prec, *default)
        assert cloudsc.get_schedule(prec) == default
        cloudsc.set_schedule(prec, 1, 448, 0)
        assert cloudsc.get_schedule(prec) == (1, 448, 0)
        cloudsc.set_schedule(prec, *default)
        assert cloudsc.get_schedule(prec) == default
    with pytest.raises(cloudsc.CloudscError):
        cloudsc.set_schedule(cloudsc.FP64, 1, 0, 2)
    with pytest.raises(cloudsc.CloudscError):
        cloudsc.set_launch(cloudsc.FP64, 0, 0)


def test_tune_picks_fastest_and_caches(tmp_path, restore_schedule):
    cache = str(tmp_path / "sched.json")
    cands = autotune.candidates(cloudsc.FP64)
    target = cands[len(cands) // 2]
    seen = []

    def timer(s):
        seen.append(s)
        return 1.0 if s == target else 2.0 + 0.01 * len(seen)

    before = cloudsc.get_schedule(cloudsc.FP64)
    r = autotune.tune(None, None, 128, 137, 2048, 262144, 3600.0, cloudsc.FP64, cache=cache, timer=timer,
                      device_name="fake")
    assert seen == cands
    assert cloudsc.get_schedule(cloudsc.FP64) == target
    assert r["best"]["ms"] == 1.0 and len(r["trials"]) == len(cands)
    data = json.load(open(cache))
    assert list(data) == ["fake|fp64|128x137x2048"]
    # applying the cached entry restores the tuned schedule
    cloudsc.set_schedule(cloudsc.FP64, *before)
    e = autotune.apply_cached(cloudsc.FP64, 128, 137, 2048, cache=cache, device_name="fake")
    assert e is not None and cloudsc.get_schedule(cloudsc.FP64) == target
    assert autotune.apply_cached(cloudsc.MIXED, 128, 137, 2048, cache=cache, device_name="fake") is None
    assert autotune.apply_cached(cloudsc.FP64, 64, 137, 2048, cache=cache, device_name="fake") is None


def test_tune_restores_schedule_on_error(tmp_path, restore_schedule):
    before = cloudsc.get_schedule(cloudsc.MIXED)

    def timer(s):
        raise RuntimeError("timer failed")

    with pytest.raises(RuntimeError):
        autotune.tune(None, None, 128, 137, 4, 512, 3600.0, cloudsc.MIXED, cache=None, timer=timer,
                      device_name="fake")
    assert cloudsc.get_schedule(cloudsc.MIXED) == before


def test_fallback_columns_take_the_choice_by_size(restore_schedule, monkeypatch):
    """The surrogate's FP64 fallback runs its few columns by size, whatever
    schedule is set for full-size calls, and leaves the thread and the set
    schedule as it found them, also when the call raises."""
    from openifs_b200 import surrogate
    L, seen = cloudsc.lib(), []

    def by_size():
        on = L.cloudsc_b200_schedule_by_size(0)
        L.cloudsc_b200_schedule_by_size(on)
        return on

    def call(*args, **kw):
        seen.append(by_size())
        if len(seen) == 2:
            raise RuntimeError("launch failed")

    monkeypatch.setattr(cloudsc, "cloudsc_batched", call)
    r = surrogate.Runner.__new__(surrogate.Runner)
    r.params, r.compact, r.nproma, r.cap, r.ptsphy = None, {}, 128, 3072, 3600.0
    cloudsc.set_schedule(cloudsc.FP64, 2, 384, 0)
    assert by_size() == 0
    r._fallback(None)
    assert by_size() == 0
    with pytest.raises(RuntimeError):
        r._fallback(None)
    assert by_size() == 0 and seen == [1, 1]
    with cloudsc.schedule_by_size(), cloudsc.schedule_by_size():
        assert by_size() == 1
    assert by_size() == 0
    assert cloudsc.get_schedule(cloudsc.FP64) == (2, 384, 0)
