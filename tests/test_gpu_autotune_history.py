"""The autotuner's times do not depend on what the set has run before, nor on
the trials before: a candidate of one cycle per launch runs one cycle per
launch, although a set past 256 cycles takes longer graphs by itself.  (A graph
captured and instantiated inside a trial of four cycles makes it three times
as long or more.)  Tuning does not count as cycles of the set either."""
import statistics

import pytest

pytestmark = pytest.mark.gpu


def _times(lulesh, before, rounds):
    with lulesh.LuleshSet.batch([lulesh.JobSpec(24), lulesh.JobSpec(28)]) as s:
        s.step(before)
        s.sync()
        rec = s.autotune(trial_cycles=4, rounds=rounds)
        assert s.state()["cycle"] == before
        return [t["ms_per_cycle"] for t in rec["trials"] if t["graph_cycles"] == 1]


def test_trials_after_a_long_run(lulesh):
    fresh = statistics.median(_times(lulesh, 3, 2))
    assert statistics.median(_times(lulesh, 300, 2)) < 1.35 * fresh


def test_trials_of_a_long_search(lulesh):
    # 18 shapes x 5 cycles x 5 rounds: 256 cycles pass in the third round; the
    # last trial of one cycle per launch is the winning shape's second one
    ms = _times(lulesh, 3, 5)
    assert ms[-1] < 1.35 * min(ms[:-1])
