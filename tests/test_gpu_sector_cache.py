"""The pair cache under sector periodicity: a body that is turned back into the
sector in the very step that builds the lists meets its new neighbours in the
next one, against the CPU oracle."""
import numpy as np
import pytest

from conftest import canonical, keys, rel_err
from fundem_b200 import scenario as S
import parity_cases as PC

pytestmark = pytest.mark.gpu


def _scene():
    sc = PC.sector()
    P = sc.particles
    pitch = sc.domain_max[0] / 4
    # body 0 crosses the x face in the first step and comes back through the
    # y face, onto body 1.  It is above the domain before and after, and the
    # two are alone, so that nothing else asks for new lists
    sc.particles = P = S.Objects(*(np.array(getattr(P, k)[:2]) for k in ("pos", "vel", "angvel", "quat", "mat", "geo")))
    P.pos[:] = [[1e-7, 1.5 * pitch, 2.4 * pitch], [2.45 * pitch, 0.1 * pitch, 2.38 * pitch]]
    sc.domain_max[2] = 2.39 * pitch
    P.vel[:] = [[-0.2, 0.0, 0.0], [0.0, 0.0, 0.0]]
    P.angvel[:] = 0.0
    return sc


def _owners(sc, contacts):
    base = np.concatenate([[0], np.cumsum([len(sc.particle_geometries[g].nodes) for g in sc.particles.geo])])
    return np.searchsorted(base, contacts["master"], side="right") - 1


def test_a_turned_body_meets_its_new_neighbours(fundem, oracle_mod):
    sc = _scene()
    g, o = fundem.Simulation.from_scenario(sc), oracle_mod.OracleWorld.from_scenario(sc)
    g.set_pair_cache(1)
    g.detect()
    o.initial_detect()
    met = []
    for _ in range(4):
        g.step(1)
        o.step(1)
        c = o.contacts(0)
        met.append(int(np.sum((_owners(sc, c) == 0) & (c["slave"] == 1))))
        assert np.array_equal(keys(canonical(g.contacts(0))), keys(canonical(c)))
        assert rel_err(g.state()["force"], o.state()["force"]) < 1e-10
    assert met[0] == 0 and met[1] > 0, met
    assert g.pair_cache_stats()[0] < 4  # some of the steps kept their lists
    g.sync()
    g.close()
