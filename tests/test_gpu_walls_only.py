"""Walls move in steps of a simulation without particles as they do beside them."""
import numpy as np
import pytest

from fundem_b200 import scenario as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form", ["step", "graph", "hook"])
@pytest.mark.parametrize("particles", [0, 1])
def test_walls_move_without_particles(fundem, particles, form):
    n, v, w = 7, np.array([0.3, -0.2, 0.1]), np.array([0.0, 0.0, 50.0])
    wg, walls = S.box_walls(np.zeros(3), np.ones(3) * 0.1, faces=("+z", "-z"))
    z3 = np.zeros((particles, 3))
    objs = S.Objects(z3 + 0.05, z3.copy(), z3.copy(), np.tile([1.0, 0, 0, 0], (particles, 1)),
                     np.zeros(particles, np.int32), np.zeros(particles, np.int32))
    sc = S.Scenario(domain_min=-0.05 * np.ones(3), domain_max=0.15 * np.ones(3), gravity=np.zeros(3), dt=1e-4,
                    particle_materials=[(1e4, 8e3, 0.5, 0.4)], wall_materials=[(0.4, 0.4)],
                    particle_geometries=[S.sphere_template(1e-3, mass=1e-5, inertia=[4e-12] * 3 + [0] * 3)] * particles,
                    wall_geometries=wg, particles=objs, walls=walls, wall_motion=[(1, v, w)])
    s = fundem.Simulation.from_scenario(sc)
    s.detect()
    at = s.state(wall=True)
    if form == "hook":
        for _ in range(n):
            s.step_begin()
            s.step_end()
    else:
        (s.step_graph if form == "graph" else s.step)(n)
    s.sync()
    st = s.state(wall=True)
    assert np.allclose(st["pos"][1], at["pos"][1] + n * sc.dt * v, rtol=0, atol=1e-15)
    assert np.array_equal(st["pos"][0], at["pos"][0]) and np.array_equal(st["quat"][0], at["quat"][0])
    # turned by n dt |w| about z
    q0, q1 = at["quat"][1], st["quat"][1]
    turn = 2.0 * np.arccos(np.clip(abs(np.dot(q0, q1)), 0.0, 1.0))
    assert abs(turn - n * sc.dt * np.linalg.norm(w)) < 1e-6
    s.close()
