"""Periodicity switched between steps, without a setup: the image sets stay
those of the last setup, a direction switched off is not detected any more,
and one switched on has no images before the next setup.  Staged steps, with
and without the pair cache, plain and from a graph; bit for bit against
simulations that never had the other flags."""
import copy

import numpy as np
import pytest

from conftest import canonical, keys
import parity_cases as PC

pytestmark = pytest.mark.gpu


def _sim(fundem, sc, flags, cache):
    sc = copy.deepcopy(sc)
    sc.periodic_x, sc.periodic_y, sc.periodic_sector = flags
    s = fundem.Simulation.from_scenario(sc)
    s.set_neighbour_list(1)  # the staged kernels at this size
    s.set_pair_cache(cache)
    return s


def _go(s, form, n):
    (s.step_graph if form == "graph" else s.step)(n)
    s.sync()


def _same(a, b, kinds):
    x, y = a.state(), b.state()
    for k in x:
        assert np.array_equal(x[k], y[k]), k
    for k in kinds:
        p, q = canonical(a.contacts(k)), canonical(b.contacts(k))
        assert np.array_equal(keys(p), keys(q)), k
        assert np.array_equal(p["spring"], q["spring"]), k


def _hand_over(a, b, kinds):
    b.set_state(**a.state())
    b.set_state(wall=True, **a.state(wall=True))
    for k in kinds:
        c = a.contacts(k)
        b.set_contacts(k, c["master"], c["slave"], c["spring"])
    if len(a.bonds()["activated"]):
        b.set_bond_activation(a.bonds()["activated"])


FORMS = pytest.mark.parametrize("form", ["step", "graph"])
CACHE = pytest.mark.parametrize("cache", [0, 1])


@FORMS
@CACHE
@pytest.mark.parametrize("before,after,kinds", [((1, 1, 0), (0, 0, 0), (0, 1)), ((0, 0, 1), (0, 0, 0), (0, 1)),
                                                ((1, 0, 1), (1, 0, 0), (0, 1, 2)), ((1, 1, 1), (0, 0, 0), (0, 1))])
def test_switched_off(fundem, before, after, kinds, cache, form):
    sc = PC.sector() if before[2] else PC.periodic()
    a, b = _sim(fundem, sc, before, cache), _sim(fundem, sc, after, cache)
    a.detect()
    _go(a, form, 2)
    a.set_periodic(*after[:2])
    a.set_periodic_sector(after[2])
    _hand_over(a, b, kinds)
    for _ in range(2):
        _go(a, form, 2)
        _go(b, form, 2)
        _same(a, b, kinds)
    a.close()
    b.close()


@FORMS
@CACHE
@pytest.mark.parametrize("flags", [(1, 0, 0), (1, 1, 0), (0, 0, 1)])
def test_switched_on(fundem, flags, cache, form):
    """Bodies inside the domain: nothing changes before a setup, and after one
    the run is that of a simulation with the flags from the start."""
    sc = PC.cluster()
    a, b = _sim(fundem, sc, (0, 0, 0), cache), _sim(fundem, sc, (0, 0, 0), cache)
    for s in (a, b):
        s.detect()
        _go(s, form, 2)
    a.set_periodic(*flags[:2])
    a.set_periodic_sector(flags[2])
    for s in (a, b):
        _go(s, form, 3)
        s.detect()
    _same(a, b, (0, 1))
    c = _sim(fundem, sc, flags, cache)
    _hand_over(a, c, (0, 1))
    a.setup(sc.domain_min, sc.domain_max)
    for s in (a, c):
        s.detect()
        _go(s, form, 3)
    _same(a, c, range(8))
    for s in (a, b, c):
        s.close()
