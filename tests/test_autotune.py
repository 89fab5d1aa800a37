"""The tuner's cache and candidates, with the library's calls and the clock replaced
(what it times on a GPU is the caller's business)."""
import json

import pytest

import autotune

SHAPE = dict(trace_len=1 << 20, width=379, expansion=4)


@pytest.fixture
def fake(monkeypatch, tmp_path):
    """A tuner on a machine without a GPU: records the knobs set; every candidate takes 1 s."""
    import torch

    class Fake:
        path = str(tmp_path / "tuning.json")
        set = []
        timed = 0

    f = Fake()
    f.set = []

    def timed(fn, reps=3):
        f.timed += 1
        return 1.0

    monkeypatch.setattr(autotune.tvmc, "set_tuning", lambda k, v: f.set.append((k, v)))
    monkeypatch.setattr(autotune, "_time", timed)
    monkeypatch.setattr(autotune, "_device_name", lambda: "gpu")
    monkeypatch.setattr(torch, "empty", lambda *a, **k: torch.zeros(1))
    lib = tmp_path / "lib.so"
    lib.write_bytes(b"one build")
    monkeypatch.setattr(autotune.tvmc, "LIB_PATH", str(lib))
    f.lib = lib
    autotune._build.cache_clear()
    yield f
    autotune._build.cache_clear()


def tune(f, **kw):
    f.set.clear()
    f.timed = 0
    return autotune.tune_commit(0, path=f.path, **SHAPE, **kw)


def test_a_choice_is_kept_for_the_same_build_only(fake):
    first = tune(fake)
    assert fake.timed > 0
    assert tune(fake) == first and fake.timed == 0 and dict(fake.set) == first["knobs"]
    fake.lib.write_bytes(b"another build")
    autotune._build.cache_clear()
    tune(fake)
    assert fake.timed > 0


def test_entries_without_a_build_are_not_applied(fake):
    old = {"knobs": {"lde_mid_variant": 2}, "seconds": {}}
    with open(fake.path, "w") as fp:
        json.dump({"gpu|commit|1048576x379x4": old}, fp)
    assert tune(fake) != old and fake.timed > 0


def test_only_knobs_that_do_something_are_timed(fake):
    entry = tune(fake)
    assert set(entry["knobs"]) == {"lde_mid_variant", "lde_mid_ctas", "lde_split_l1", "ntt_tile_log"}
    assert "hash_unfused_tree" not in dict(fake.set)


@pytest.mark.parametrize("log_n", [8, 12, 13, 16, 17, 20, 22])
def test_candidates_are_valid_and_distinct(log_n):
    c = autotune.lde_candidates(log_n)
    balanced = (log_n + 1) // 2
    assert len({tuple(x.items()) for x in c}) == len(c)
    for x in c:
        s = x["lde_split_l1"]
        assert s == 0 or (6 <= s <= 12 and 6 <= log_n - s <= 12)
        if x["lde_mid_variant"] == 0:
            assert x["lde_mid_ctas"] == 3
        else:
            assert s != balanced  # the networks' default
    if log_n >= 12:
        assert any(x["lde_mid_variant"] == 0 and x["lde_split_l1"] == balanced for x in c)
    assert {x["lde_mid_variant"] for x in c if x["lde_split_l1"] == 0} == {0, 1, 2}
