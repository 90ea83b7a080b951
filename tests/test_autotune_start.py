"""The autotuner's search starts from the slices that the engine takes by itself and never
ends with ones that it timed slower (a fake engine whose throughput is a table)."""
import pytest

from hawassi_c_b200 import autotune

NXS = {"a": 2048, "b": 4096}
RATE = {(512, 512): 9.0, (1024, 512): 5.0, (2048, 512): 4.0, (512, 1024): 6.0, (512, 2048): 5.0, (2048, 2048): 7.0,
        (2048, 1024): 6.5, (1024, 2048): 6.0, (1024, 1024): 5.5}


class FakeEngine:
    clock = 0.0

    def __init__(self, decks, slices=None, **kw):
        self.members = len(decks)
        self.slices = [512 if slices is None else slices[NXS[d]] for d in decks]
        self.calls = 0

    def run(self, i_stop, sync=True):
        self.calls += 1
        FakeEngine.clock += 1.0 / RATE[tuple(self.slices)]

    def stats(self, m):
        return {"rhs_calls": self.calls}

    def close(self):
        pass


def test_starts_from_the_engines_choice(monkeypatch):
    monkeypatch.setattr(autotune, "Engine", FakeEngine)
    monkeypatch.setattr(autotune, "deck_table", lambda d, name: [NXS[d]])
    monkeypatch.setattr(autotune.time, "perf_counter", lambda: FakeEngine.clock)
    best, trials = autotune.autotune_slices(["a", "b"], window=3, warm=1)
    assert trials[0][0] == {2048: 512, 4096: 512}
    assert best == {2048: 512, 4096: 512}
    assert dict((tuple(t.values()), v) for t, v in trials)[(512, 512)] == pytest.approx(max(v for _, v in trials))
