"""Sums of the pairs' forces: pairs of a few contacts and of hundreds (bodies
pressed into one another), more and fewer pairs than a warp takes, in staged
and small steps, against the CPU oracle.  The order is the
contacts', so every launch shape gives the same bits."""
import numpy as np
import pytest

from conftest import canonical, keys, rel_err
from fundem_b200 import scenario as S

pytestmark = pytest.mark.gpu


def _pressed(n, gap):
    """n pairs of spheres, the pairs apart from one another, the two of a pair
    `gap` radii between their centres."""
    r = 1e-3
    geo = S.sphere_template(r, level=3, mass=1e-5, inertia=[4e-12] * 3 + [0] * 3)
    side = int(np.ceil(n ** (1 / 3)))
    g = np.arange(side) * 5e-3
    X, Y, Z = np.meshgrid(g, g, g)
    c = np.stack([X.ravel(), Y.ravel(), Z.ravel()], 1)[:n]
    pos = np.concatenate([c, c + np.array([gap * r, 0, 0])])
    rng = np.random.default_rng(n)
    m = 2 * n
    objs = S.Objects(pos, rng.uniform(-0.1, 0.1, (m, 3)), np.zeros((m, 3)), S.random_quaternions(rng, m),
                     np.zeros(m, np.int32), np.zeros(m, np.int32))
    return S.Scenario(domain_min=-5e-3 * np.ones(3), domain_max=(side + 1) * 5e-3 * np.ones(3), gravity=np.zeros(3),
                      dt=1e-7, particle_materials=[(1e4, 8e3, 0.5, 0.4)], wall_materials=[(0.4, 0.4)],
                      particle_geometries=[geo], wall_geometries=[], particles=objs, walls=S.Objects.empty())


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("n,gap", [(1, 1.95), (1, 0.3), (3, 0.3), (33, 0.3), (33, 1.6), (700, 0.5)])
def test_pair_sums_of_few_and_many_contacts(fundem, oracle_mod, n, gap, precision):
    sc = _pressed(n, gap)
    runs = []
    for staged, shape in ((False, (0, 0, 0, 0)), (True, (0, 0, 0, 0)), (True, (1, 1, 1, 1)), (True, (8, 8, 8, 16))):
        s = fundem.Simulation.from_scenario(sc, precision=precision)
        s.set_neighbour_list(1 if staged else 0)
        s.set_launch_shape(*shape)
        s.detect()
        s.step(2)
        s.sync()
        runs.append((s.state(), s.contacts(fundem.PP)))
        s.close()
    st, c = runs[0]
    assert len(c["master"]) >= (1 if gap > 1 else 150) * n
    for other, _ in runs[1:]:
        for k in ("force", "torque", "pos", "vel"):
            assert np.array_equal(other[k], st[k]), k
    if precision == 0:
        o = oracle_mod.OracleWorld.from_scenario(sc)
        o.initial_detect()
        o.step(2)
        assert np.array_equal(keys(canonical(c)), keys(canonical(o.contacts(0))))
        for k in ("force", "torque"):
            assert rel_err(st[k], o.state()[k]) < 1e-10, k
