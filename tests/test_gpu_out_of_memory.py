"""Calls that find no device memory fail with an error, and work once there is
some: an array whose allocation failed is empty, not there without memory."""
import numpy as np
import pytest

from conftest import canonical
from fundem_b200 import scenario as S
import parity_cases as PC

pytestmark = pytest.mark.gpu


class Hold:
    """All device memory but `leave` bytes, while it lasts."""

    def __init__(self, leave):
        self.leave = leave

    def __enter__(self):
        import torch
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        self.block = torch.empty(torch.cuda.mem_get_info()[0] - self.leave, dtype=torch.uint8, device="cuda")

    def __exit__(self, *_):
        import torch
        del self.block
        torch.cuda.empty_cache()


def test_adjoint_tape(fundem):
    sc = PC.pour_mm(n=64)
    rng = np.random.default_rng(3)
    w, u = rng.standard_normal((2, 64, 3))

    def run(tight):
        s = fundem.Simulation.from_scenario(sc, records=False)
        s.detect()
        s.adjoint_begin(2000)       # a tape of 2,000 steps: some 400 MB
        s.adjoint_forward(20)
        s.sync()
        if tight:
            for _ in range(2):
                with Hold(100 << 20):
                    with pytest.raises(fundem.FundemError):
                        s.adjoint_backward(w, u)
        out = s.adjoint_backward(w, u)
        s.adjoint_end()
        s.step(1)
        s.sync()
        s.close()
        return out

    ref, got = run(False), run(True)
    for a, b in zip(ref, got):
        assert np.abs(a - b).max() <= 1e-12 * np.abs(a).max()   # the sweep adds with atomics


def _boxes(n):
    """Boxes of 17 x 17 nodes a face lying on a floor: 289 contacts each."""
    m, G = 17, 32
    a, b = (v.ravel() for v in np.meshgrid(*[np.linspace(-1e-3, 1e-3, m)] * 2))
    faces = [np.roll(np.stack([np.full(m * m, side), a, b], 1), d, 1) for d in range(3) for side in (-1e-3, 1e-3)]
    ax = np.linspace(-1.3e-3, 1.3e-3, G)
    q = np.abs(np.stack(np.meshgrid(ax, ax, ax, indexing="ij")[::-1], -1)) - 1e-3
    sdf = np.linalg.norm(np.maximum(q, 0), axis=-1) + np.minimum(q.max(-1), 0)
    geo = S.Geometry(origin=np.full(3, ax[0]), spacing=ax[1] - ax[0], size=np.array([G] * 3, np.int32),
                     sdf=sdf.reshape(-1).copy(), nodes=np.unique(np.concatenate(faces).round(9), axis=0),
                     tris=np.zeros((0, 3), np.int32), mass=2e-5, inertia=np.array([1.3e-11] * 3 + [0.0] * 3))
    side = int(np.ceil(n ** 0.5))
    i = np.arange(n)
    pos = np.stack([(i % side + 0.5) * 2.05e-3, (i // side + 0.5) * 2.05e-3, np.full(n, 1e-3 - 1e-7)], 1)
    z3 = np.zeros((n, 3))
    objs = S.Objects(pos, z3, z3.copy(), np.tile([1.0, 0, 0, 0], (n, 1)), np.zeros(n, np.int32), np.zeros(n, np.int32))
    box = np.array([side * 2.05e-3, side * 2.05e-3, 6e-3])
    wg, w = S.box_walls(np.zeros(3), box)
    return S.Scenario(domain_min=-2e-3 * np.ones(3), domain_max=box + 2e-3, gravity=np.array([0, 0, -9.81]), dt=1e-6,
                      particle_materials=[(1e4, 8e3, 0.5, 0.4)], wall_materials=[(0.4, 0.4)],
                      particle_geometries=[geo], wall_geometries=wg, particles=objs, walls=w)


@pytest.mark.parametrize("staged", [False, True])
@pytest.mark.parametrize("n", [1000, 2500])   # 30 MB of contacts, which the read-back keeps room for, and 75, which it gives back
def test_contacts_read_without_device_memory(fundem, n, staged):
    import torch
    s = fundem.Simulation.from_scenario(_boxes(n))
    s.set_neighbour_list(1 if staged else 0)
    s.detect()
    s.step(2)
    s.sync()
    free = torch.cuda.mem_get_info()[0]
    with Hold(16 << 20):
        tight = canonical(s.contacts(fundem.PW))
    roomy = canonical(s.contacts(fundem.PW))
    assert len(roomy["master"]) >= 289 * n
    for k in roomy:
        assert np.array_equal(roomy[k], tight[k]), k
    assert free - torch.cuda.mem_get_info()[0] <= 64 << 20
    s.step(1)
    s.sync()
    s.close()
