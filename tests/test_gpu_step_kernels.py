"""Branches of the step kernels that ordinary scenes rarely reach, GPU engine against the oracle, bit for bit
(the exact variant runs the oracle's IEEE operations in its order, so the tolerance is zero; orientations 1e-12
as everywhere)."""
import numpy as np
import pytest

from oracle import bridge
from woo_gb300 import abi, scenes

from helpers import assert_same_contacts, assert_same_particles, gpu_handle, gpu_particles

pytestmark = pytest.mark.gpu


def _run_both(spec, steps):
    h = gpu_handle(spec)
    o = bridge.Oracle(spec.params, spec.particles, cell=spec.cell)
    for k in steps:
        h.step(k)
        o.step(k)
        assert_same_particles(gpu_particles(h, spec.particles.n), o.particles())
        assert_same_contacts(h.download_contacts(), o.contacts())
    return h, o


@pytest.mark.parametrize("law", ["frict", "hertz"])
def test_periods_beyond_the_neighbour_cell(wdem_lib, law):
    """Contact.cellDist of several periods per axis: spheres moved by whole lattice vectors of the cell, so that the
    image shift hSize * cellDist takes its general product and not the one for 0 and +-1."""
    spec = scenes.periodic_cloud(300, 3, size=(0.08, 0.08, 0.08), law=law, shear=0.25)
    rng = np.random.default_rng(1)
    spec.particles.pos += rng.integers(-3, 4, (spec.particles.n, 3)) @ np.asarray(spec.cell["hSize"]).T
    h, o = _run_both(spec, (1, 20))
    c = h.download_contacts()
    assert (np.abs(c.cellDist[c.real == 1]) > 1).any()


def test_hertz_materials_with_alpha(wdem_lib):
    """HertzMat.alpha != 0 (without surface energy): the noAttraction clamp does not apply to those contacts."""
    spec = scenes.random_cloud(300, 4, dense=0.8, law="hertz")
    for k in range(2):
        spec.materials[k].surfEnergy = 0.0
    spec.materials[1].alpha = 0.4
    h, _ = _run_both(spec, (1, 60))
    assert h.status().nReal > 50


@pytest.mark.parametrize("m", [63, 64, 65, 96, 97, 200])
def test_wall_force_over_long_rows(wdem_lib, m):
    """The force on a wall from m spheres touching it, and as many hovering above: rows at and beyond the length
    where a warp takes them from the single thread, with stamped and unstamped records mixed."""
    r = 0.005
    k = np.arange(2 * m)
    side = int(np.ceil(np.sqrt(2 * m)))
    centers = np.stack([0.02 + 2.2 * r * (k % side), 0.02 + 2.2 * r * (k // side), np.where(k % 2, 1.02 * r, 0.98 * r)], axis=1)
    mats = [dict(kind=abi.MAT_FRICT, density=2500.0, young=1e7, ktDivKn=0.2, tanPhi=0.5)]
    pa = scenes.assemble(centers, np.full(2 * m, r), 0, [(2, 1, 0.0, 0)], mats, vel=np.random.default_rng(m).normal(0, 0.2, (2 * m, 3)))
    spec = scenes.SceneSpec(scenes.default_params(scenes.materials_array(mats), dt=1e-5, gravity=(0, 0, -9.81)), None, pa)
    h, _ = _run_both(spec, (1, 3))
    assert h.status().nReal >= m
