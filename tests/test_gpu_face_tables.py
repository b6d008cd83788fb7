"""The tables of cell faces are a copy of the SDF grids that saves loads: with
little device memory free a run goes without them, and gives the same bits."""
import numpy as np
import pytest

from conftest import canonical, keys
from fundem_b200 import scenario as S

pytestmark = pytest.mark.gpu

GRID = 96                     # points an axis: 15 MB of double values, tables of 42 MB
TABLES = 48 * GRID ** 3


def _heap():
    n = 64
    rng = np.random.default_rng(4)
    geo = S.superellipsoid_templates(rng, 1, n=GRID, level=2, explicit_mass=True)
    box = 4 * 2.05e-3 * np.ones(3)
    pos = S.lattice_positions(rng, n, np.zeros(3), box + 1e-12, 2.05e-3, 2e-5)
    objs = S.Objects(pos, rng.uniform(-0.05, 0.05, (n, 3)), np.zeros((n, 3)), S.random_quaternions(rng, n),
                     np.zeros(n, np.int32), np.zeros(n, np.int32))
    wg, w = S.box_walls(np.zeros(3), box)
    return S.Scenario(domain_min=-2e-3 * np.ones(3), domain_max=box + 2e-3, gravity=np.array([0, 0, -9.81]), dt=1e-6,
                      particle_materials=[(1e4, 8e3, 0.5, 0.4)], wall_materials=[(0.4, 0.4)], particle_geometries=geo,
                      wall_geometries=wg, particles=objs, walls=w)


def _run(fundem, torch, sc, precision, staged):
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    s = fundem.Simulation.from_scenario(sc, precision=precision)
    used = before - torch.cuda.mem_get_info()[0]
    s.set_neighbour_list(1 if staged else 0)
    s.detect()
    s.step(4)
    s.sync()
    out = s.state(), canonical(s.contacts(fundem.PP)), canonical(s.contacts(fundem.PW))
    s.close()
    return used, out


@pytest.mark.parametrize("staged", [False, True])
@pytest.mark.parametrize("precision", [0, 1])
def test_runs_without_the_tables(fundem, precision, staged):
    import torch
    sc = _heap()
    _run(fundem, torch, sc, precision, staged)   # what the first run loads stays
    used, ref = _run(fundem, torch, sc, precision, staged)
    hold = torch.empty(torch.cuda.mem_get_info()[0] - (250 << 20), dtype=torch.uint8, device="cuda")
    try:
        tight, got = _run(fundem, torch, sc, precision, staged)
    finally:
        del hold
        torch.cuda.empty_cache()
    if precision == 0:
        assert used - tight > 0.9 * TABLES
    for k in ref[0]:
        assert np.array_equal(ref[0][k], got[0][k]), k
    for a, b in zip(ref[1:], got[1:]):
        assert np.array_equal(keys(a), keys(b))
        assert len(a["master"]) > 0
        for k in ("overlap", "normal", "spring"):
            assert np.array_equal(a[k], b[k]), k


def test_tables_of_a_changed_precision(fundem):
    """Set up in mixed precision, stepped in double: before and after the next
    setup the bits of a run that was in double from the start."""
    sc = _heap()
    ref = fundem.Simulation.from_scenario(sc)
    s = fundem.Simulation.from_scenario(sc, precision=fundem.FP32_MIXED)
    s.set_precision(fundem.FP64)
    for again in range(2):
        for g in (ref, s):
            if again:
                g.setup(sc.domain_min, sc.domain_max)
            g.detect()
            g.step(3)
            g.sync()
        a, b = ref.state(), s.state()
        for k in a:
            assert np.array_equal(a[k], b[k]), k
    ref.close()
    s.close()
