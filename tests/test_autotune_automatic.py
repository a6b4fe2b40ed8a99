"""The automatic choices are candidates wherever they run kernels of their
own (windows asked for turn off the pancake windows of 8! states and, as
asked-for threads and far marks do, the one-launch search), so that a tuned
search is never slower than an untuned one.  The searches are faked."""
import pytest

from puzzlesearch_b200 import autotune


class Fake:
    """bfs() of a puzzle whose automatic search takes 1 ms, in one launch or
    (whole=False) level by level, and 2 ms and more with anything asked for."""

    def __init__(self, monkeypatch, whole=True):
        self.calls, self.whole = [], whole
        monkeypatch.setattr(autotune, "bfs", self.bfs)
        monkeypatch.setattr(autotune, "device_name", lambda: "GPU")

    def bfs(self, puzzle, algo, initial=0, max_depth=0, window_bits=0, direction="auto", far_marks="auto", threads=0):
        self.calls.append((window_bits, far_marks, threads))
        asked = bool(window_bits) or far_marks != "auto" or bool(threads)
        ms = 1.0 if not asked else 2.0 + window_bits / 100 + threads / 1000
        levels = 9
        return {"counts": [1, 2, 3], "stats": {"total_ms": ms, "window_bits": 16, "levels": levels,
                                               "expand_launches": 1 if self.whole and not asked else levels}}


@pytest.mark.parametrize("whole", [True, False])
def test_window_bits(monkeypatch, whole):
    Fake(monkeypatch, whole)
    best, timings = autotune.tune_window_bits(None, "two_bit")
    assert best == 0 and set(timings) == {0, 14, 15, 16, 17, 18}


def test_threads_and_far_marks_of_one_launch_searches(monkeypatch):
    Fake(monkeypatch)
    best, timings = autotune.tune_threads(None, "two_bit")
    assert best == 0 and set(timings) == {0, 128, 256, 512}
    best, timings = autotune.tune_far_marks(None)
    assert best == "auto" and set(timings) == {"auto", "none", "near", "all"}


def test_threads_and_far_marks_level_by_level(monkeypatch):
    """The automatic choice is one of the others there; nothing to add."""
    Fake(monkeypatch, whole=False)
    assert set(autotune.tune_threads(None, "two_bit")[1]) == {128, 256, 512}
    assert set(autotune.tune_far_marks(None)[1]) == {"none", "near", "all"}


TUNERS = [(lambda c: autotune.tune_window_bits(None, "two_bit", cache=c, key="w"), 0, 16),
          (lambda c: autotune.tune_threads(None, "two_bit", cache=c, key="w"), 0, 256),
          (lambda c: autotune.tune_far_marks(None, cache=c, key="w"), "auto", "near")]


@pytest.mark.parametrize("tuner,automatic,other", TUNERS, ids=["window_bits", "threads", "far_marks"])
def test_cached_picks(monkeypatch, tmp_path, tuner, automatic, other):
    """The automatic choice is cached like any other; a pick made without it
    among the candidates is made again."""
    fake = Fake(monkeypatch)
    path = str(tmp_path / "tune.json")
    assert tuner(autotune.Cache(path))[0] == automatic
    n = len(fake.calls)
    assert tuner(autotune.Cache(path)) == (automatic, {}) and len(fake.calls) == n
    old = autotune.Cache(str(tmp_path / "old.json"))
    old.put("GPU", "w", other)
    assert tuner(old)[0] == automatic and old.get("GPU", "w") == automatic


def test_candidates_asked_for(monkeypatch):
    """Only those are timed, and a cached pick of theirs is taken as it is."""
    Fake(monkeypatch)
    cache = autotune.Cache(None)
    assert set(autotune.tune_window_bits(None, "two_bit", candidates=[12, 14])[1]) == {12, 14}
    assert set(autotune.tune_threads(None, "two_bit", candidates=(128, 512))[1]) == {128, 512}
    cache.put("GPU", "w", 14)
    assert autotune.tune_window_bits(None, "two_bit", candidates=[12, 14], cache=cache, key="w") == (14, {})
