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
