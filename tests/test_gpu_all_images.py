"""Translated and turned images in one run: with x, y and sector periodicity a
step has eight contact lists, six of them of images, against the CPU oracle.
The turned images' last bits may differ (CUDA's sines and cosines, the host
library's), so the pairs are compared exactly and the numbers to the
tolerances of the sector tests."""
import numpy as np
import pytest

from conftest import canonical, keys, rel_err
import parity_cases as PC

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cache", [0, 1])
@pytest.mark.parametrize("x,y", [(True, False), (False, True), (True, True)])
def test_sector_with_translated_images_vs_oracle(fundem, oracle_mod, x, y, cache):
    sc = PC.sector()
    sc.periodic_x, sc.periodic_y = x, y
    g, o = fundem.Simulation.from_scenario(sc), oracle_mod.OracleWorld.from_scenario(sc)
    g.set_pair_cache(cache)
    g.detect()
    o.initial_detect()
    images = [2] * x + [3] * y + [4] * (x and y) + [5, 6, 7]
    assert all(len(o.contacts(k)["master"]) for k in images)
    for _ in range(4):
        for k in range(8):
            a, b = canonical(g.contacts(k)), canonical(o.contacts(k))
            assert np.array_equal(keys(a), keys(b)), k
            if len(b["overlap"]):
                assert rel_err(a["overlap"], b["overlap"]) < 1e-9, k
        g.step(1)
        o.step(1)
        sg, so = g.state(), o.state()
        for k, tol in (("force", 1e-10), ("torque", 1e-10), ("pos", 1e-13), ("vel", 1e-10), ("angvel", 1e-10),
                       ("quat", 1e-13)):
            assert rel_err(sg[k], so[k]) < tol, k
    g.sync()
    g.close()
