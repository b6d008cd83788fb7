"""Runs of several phases on one simulation: setup, detect, steps, and again.
Every later phase gives what a fresh simulation gives that is handed the same
state, springs and bonds, bit for bit: nothing of the staged steps' tables
(cell lists, reverse index, pair cache) outlives a setup."""
import copy

import numpy as np
import pytest

from conftest import canonical, keys
from fundem_b200 import scenario as S
import parity_cases as PC

pytestmark = pytest.mark.gpu


def heap(n, seed=1):
    """n bodies of a lattice pulled together until neighbours overlap, in a box."""
    rng = np.random.default_rng(seed)
    geos = S.superellipsoid_templates(rng, 2, n=16, level=2, explicit_mass=True)
    side = int(np.ceil(n ** (1 / 3)))
    box = side * 2.05e-3 * np.ones(3)
    pos = S.lattice_positions(rng, n, np.zeros(3), box + 1e-12, 2.05e-3, 2e-5)
    objs = S.Objects(pos, rng.uniform(-0.05, 0.05, (n, 3)), np.zeros((n, 3)), S.random_quaternions(rng, n),
                     np.zeros(n, np.int32), rng.integers(0, 2, n).astype(np.int32))
    wg, w = S.box_walls(np.zeros(3), box)
    return S.Scenario(domain_min=-2e-3 * np.ones(3), domain_max=box + 2e-3, gravity=np.array([0, 0, -9.81]), dt=1e-6,
                      particle_materials=[(1e4, 8e3, 0.5, 0.4)], wall_materials=[(0.4, 0.4)], particle_geometries=geos,
                      wall_geometries=wg, particles=objs, walls=w)


def _phase(sim, steps, form):
    sim.detect()
    if form == "graph":
        sim.step_graph(steps)
    else:
        sim.step(steps)
    sim.sync()
    bonds = sim.bonds()["activated"]
    return sim.state(), sim.state(wall=True), [canonical(sim.contacts(k)) for k in range(8)], bonds


def _fresh(fundem, sc, seen, cache):
    s = fundem.Simulation.from_scenario(copy.deepcopy(sc))
    if cache is not None:
        s.set_pair_cache(cache)
    state, walls, contacts, bonds = seen
    s.set_state(**state)
    s.set_state(wall=True, **walls)
    for k, c in enumerate(contacts):
        if len(c["master"]):
            s.set_contacts(k, c["master"], c["slave"], c["spring"])
    if len(bonds):
        s.set_bond_activation(bonds)
    return s


CASES = [("periodic", 0), ("periodic", 1), ("sector", 0), ("sector", 1), ("heap", None)]


@pytest.mark.parametrize("form", ["step", "graph"])
@pytest.mark.parametrize("steps", [1, 5])
@pytest.mark.parametrize("name,cache", CASES)
def test_a_later_phase_equals_a_fresh_simulation(fundem, name, cache, steps, form):
    sc = heap(8192) if name == "heap" else getattr(PC, name)()
    s = fundem.Simulation.from_scenario(copy.deepcopy(sc))
    if cache is not None:
        s.set_pair_cache(cache)
    seen = _phase(s, steps, form)
    for _ in range(2):
        f = _fresh(fundem, sc, seen, cache)
        s.setup(sc.domain_min, sc.domain_max)
        seen, ref = _phase(s, steps, form), _phase(f, steps, form)
        f.close()
        for a, b in ((seen[0], ref[0]), (seen[1], ref[1])):
            for k in a:
                assert np.array_equal(a[k], b[k]), k
        for k, (a, b) in enumerate(zip(seen[2], ref[2])):
            assert np.array_equal(keys(a), keys(b)), k
            for v in ("overlap", "spring", "point", "normal"):
                assert np.array_equal(a[v], b[v]), (k, v)
    assert len(seen[2][0]["master"]) > 0
    s.close()
