"""Small sets step with two launches (k_small_pairs, k_small_advance) in place
of the staged kernels; under the stage timers (fundem_set_profiling) every set
takes the staged ones.  Both sum in the same order, so a run is the same bit
for bit, whatever the count does to the blocks (four bodies each), the walls
to the lanes, or one body to its partners' list (more owners than the sum
keeps in registers)."""
import copy

import numpy as np
import pytest

from conftest import canonical, keys
from fundem_b200 import scenario as S

pytestmark = pytest.mark.gpu


def _heap(n, turning, walls=6):
    """n bodies of a lattice pulled together until neighbours overlap."""
    rng = np.random.default_rng(n)
    geos = S.superellipsoid_templates(rng, 2, n=16, level=2, explicit_mass=True)
    side = int(np.ceil(n ** (1 / 3)))
    box = side * 2.05e-3 * np.ones(3)
    pos = S.lattice_positions(rng, n, np.zeros(3), box + 1e-12, 2.05e-3, 2e-5)
    objs = S.Objects(pos, rng.uniform(-0.05, 0.05, (n, 3)), rng.uniform(-1, 1, (n, 3)) * turning,
                     S.random_quaternions(rng, n), np.zeros(n, np.int32), rng.integers(0, 2, n).astype(np.int32))
    faces = ("+z", "-z", "+x", "-x", "+y", "-y")
    wg, w = S.box_walls(np.zeros(3), box, faces=faces[:walls])
    return S.Scenario(domain_min=-2e-3 * np.ones(3), domain_max=box + 2e-3, gravity=np.array([0, 0, -9.81]), dt=1e-6,
                      particle_materials=[(1e4, 8e3, 0.5, 0.4)], wall_materials=[(0.4, 0.4)], particle_geometries=geos,
                      wall_geometries=wg, particles=objs, walls=w,
                      inertia="physical" if turning else "reference")


def _crowd(owners):
    """A large sphere, last in the order, touched by `owners` small ones."""
    small, large = S.sphere_template(1e-3, mass=1e-5, inertia=[4e-12] * 3 + [0] * 3), \
        S.sphere_template(5e-3, n=13, mass=1e-3, inertia=[1e-8] * 3 + [0] * 3)
    k = np.arange(owners) + 0.5
    phi, th = np.arccos(1 - 2 * k / owners), np.pi * (1 + 5 ** 0.5) * k
    d = np.stack([np.cos(th) * np.sin(phi), np.sin(th) * np.sin(phi), np.cos(phi)], 1)
    pos = np.concatenate([5.85e-3 * d, np.zeros((1, 3))])  # the coarse grid's surface lies up to 50 um inside
    n = owners + 1
    objs = S.Objects(pos, np.zeros((n, 3)), np.zeros((n, 3)), S.random_quaternions(np.random.default_rng(1), n),
                     np.zeros(n, np.int32), np.array([0] * owners + [1], np.int32))
    return S.Scenario(domain_min=-0.02 * np.ones(3), domain_max=0.02 * np.ones(3), gravity=np.zeros(3), dt=1e-6,
                      particle_materials=[(1e4, 8e3, 0.5, 0.4)], wall_materials=[(0.4, 0.4)],
                      particle_geometries=[small, large], wall_geometries=[], particles=objs, walls=S.Objects.empty())


def _run(fundem, sc, precision, form):
    s = fundem.Simulation.from_scenario(copy.deepcopy(sc), precision=precision)
    s.set_profiling(form == "staged")
    s.detect()
    if form == "graph":
        s.step_graph(3)
        s.step_graph(3)
    elif form == "mixed forms":
        s.step(1)
        s.set_profiling(True)   # one staged step between small ones
        s.step(1)
        s.set_profiling(False)
        s.step_begin()
        s.step_end()
        s.step_graph(3)
    else:
        s.step(6)
    s.sync()
    out = s.state(), s.state(wall=True), [canonical(s.contacts(k)) for k in (fundem.PP, fundem.PW)]
    s.close()
    return out


CASES = [("heap", n, t) for n, t in ((1, False), (3, True), (4, False), (5, True), (64, True), (343, False))]
CASES += [("heap", n, t) for n, t in ((1184, True), (1185, True), (2197, False))]  # two, then four blocks per SM
CASES += [("crowd", m, False) for m in (15, 16, 17, 40)]


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("kind,n,turning", CASES)
def test_small_steps_match_the_staged_ones(fundem, kind, n, turning, precision):
    sc = _heap(n, turning, walls=1 + n % 6) if kind == "heap" else _crowd(n)
    ref = _run(fundem, sc, precision, "staged")
    if kind == "crowd":
        assert len(np.unique(keys(ref[2][0]))) >= n
    for form in ("step", "graph", "mixed forms"):
        got = _run(fundem, sc, precision, form)
        for a, b in ((got[0], ref[0]), (got[1], ref[1])):
            for k in a:
                assert np.array_equal(a[k], b[k]), (form, k)
        for a, b in zip(got[2], ref[2]):
            assert np.array_equal(keys(a), keys(b)), form
            for k in ("overlap", "spring", "point", "normal"):
                assert np.array_equal(a[k], b[k]), (form, k)
