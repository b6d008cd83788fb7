"""Limits of the small steps.  The largest small set takes two launches a step,
one body more the staged kernels, and both give the bits of the staged form; so
does a body with more owners than one pass over its list takes (16)."""
import numpy as np
import pytest

from conftest import canonical, keys
from test_gpu_small_steps import _crowd, _heap

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [5120, 5121])
def test_the_largest_small_set(fundem, n):
    sc = _heap(n, True)
    runs = []
    for staged in (False, True):
        s = fundem.Simulation.from_scenario(sc)
        s.set_profiling(staged)
        s.detect()
        before = s.launch_count()
        s.step(4)
        s.sync()
        launches = s.launch_count() - before
        assert (launches <= 4 * 2 + 2) == (n == 5120 and not staged), launches
        runs.append((s.state(), canonical(s.contacts(fundem.PP)), canonical(s.contacts(fundem.PW))))
        s.close()
    (a, *ca), (b, *cb) = runs
    for k in a:
        assert np.array_equal(a[k], b[k]), k
    for x, y in zip(ca, cb):
        assert np.array_equal(keys(x), keys(y)) and np.array_equal(x["spring"], y["spring"])


@pytest.mark.parametrize("owners", [32, 33, 100])
def test_a_body_with_many_owners(fundem, owners):
    runs = []
    for staged in (False, True):
        s = fundem.Simulation.from_scenario(_crowd(owners))
        s.set_profiling(staged)
        s.detect()
        s.step(3)
        s.sync()
        runs.append(s.state())
        assert len(np.unique(keys(s.contacts(fundem.PP))[:, 0])) >= owners
        s.close()
    for k in runs[0]:
        assert np.array_equal(runs[0][k], runs[1][k]), k
