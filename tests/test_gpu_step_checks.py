"""The host's checks between steps (list growth every 64 steps, the pair
cache's after a forced rebuild) come before a step's first launch: a long run
in one call, which joins the halves of neighbouring steps except across the
checks, gives the bits of as many calls of one step."""
import numpy as np
import pytest

from conftest import canonical, keys
import parity_cases as PC

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name,cache", [("cluster", 0), ("cluster", 1), ("periodic", 0), ("periodic", 1)])
def test_one_call_equals_many(fundem, name, cache):
    runs = []
    for calls in ((130,), (1,) * 130, (63, 1, 2, 64)):
        s = fundem.Simulation.from_scenario(getattr(PC, name)())
        s.set_pair_cache(cache)
        s.detect()
        for k, n in enumerate(calls):
            s.step(n)
            if k == 1:
                s.set_state(vel=s.state()["vel"])   # asks for a rebuild
        s.sync()
        runs.append((s.state(), canonical(s.contacts(fundem.PP))))
        s.close()
    for st, c in runs[1:]:
        for k in st:
            assert np.array_equal(st[k], runs[0][0][k]), k
        assert np.array_equal(keys(c), keys(runs[0][1])) and np.array_equal(c["spring"], runs[0][1]["spring"])
