"""Periodic pairs of spheres many periods apart whose boxes meet within a few millionths of the cell: the reference's
test rounds min + size at the magnitude of the position and divides by it, an error of up to N M 2^-53 periods for a
body M periods out and another N periods from it.  The pairs must be those of the oracle, whose operations are the
reference's, from the neighbour cell to where that error exceeds the margin of the engine's FP32 screens (1e-6)."""
import numpy as np
import pytest

from oracle import bridge
from woo_gb300 import abi, scenes

from helpers import assert_same_contacts, gpu_handle

pytestmark = pytest.mark.gpu


def _pairs_of_spheres(periods, seed, m=6, L=0.1, r=0.003, verlet=0.0004):
    """m^3 pairs on a lattice in a cubic cell, each along one axis with a gap of +-5e-6 cell lengths between the boxes;
    every sphere moved by whole cells of its own."""
    rng = np.random.default_rng(seed)
    k = np.arange(m ** 3)
    a = (np.stack([k % m, k // m % m, k // (m * m)], axis=1) + 0.25) * (L / m) + rng.uniform(0, 0.1 * L / m, (m ** 3, 3))
    gap = 2 * (r + verlet) + rng.uniform(-5e-6, 5e-6, m ** 3) * L
    b = a + rng.uniform(0.1, 0.5, a.shape) * r
    b[k, k % 3] = a[k, k % 3] + gap
    pos = np.empty((2 * m ** 3, 3))
    pos[0::2], pos[1::2] = a, b
    pos += rng.integers(-periods, periods + 1, pos.shape) * L
    mats = [dict(kind=abi.MAT_FRICT, density=2500.0, young=1e7, ktDivKn=0.2, tanPhi=0.5)]
    ma = scenes.materials_array(mats)
    pa = scenes.assemble(pos, np.full(len(pos), r), 0, [], mats)
    p = scenes.default_params(ma, dt=1e-9, damping=0.0, verletDist=verlet)
    cell = dict(hSize=np.eye(3) * L, trsf=np.eye(3), gradV=np.zeros((3, 3)), nextGradV=np.zeros((3, 3)))
    return scenes.SceneSpec(p, ma, pa, "pairs", cell=cell)


@pytest.mark.parametrize("seed", range(3))
@pytest.mark.parametrize("periods", [1, 1000, 8191, 8192, 16383, 16384, 16385, 32768, 65536, 131072, 262144, 524288])
def test_pairs_many_periods_apart(wdem_lib, periods, seed):
    spec = _pairs_of_spheres(periods, seed)
    h = gpu_handle(spec)
    o = bridge.Oracle(spec.params, spec.particles, cell=spec.cell)
    h.step(1)
    o.step(1)
    c = o.contacts()
    assert 30 < c.n < 216
    assert_same_contacts(h.download_contacts(), c)
    assert np.array_equal(h.download_contacts().cellDist, c.cellDist)
    h.close()
