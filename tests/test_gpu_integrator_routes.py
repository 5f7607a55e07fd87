"""The integrator's two routes for spheres: one launch (scenes of up to 256 bodies an SM with the default launch shape)
and two passes (larger scenes, and every other launch shape).  Both evaluate the same expressions per particle in the
same order, so their states are equal bit for bit in each arithmetic; the exact one is the oracle's."""
import numpy as np
import pytest

from oracle import bridge
from woo_gb300 import abi, scenes

from helpers import assert_same_contacts, assert_same_particles, gpu_handle, gpu_particles
from test_gpu_fma import _handle

pytestmark = pytest.mark.gpu

TWO_PASS = [dict(integratorBlock=128, listsPerSM=1), dict(integratorBlock=512, listsPerSM=2),
            dict(integratorBlock=256, listsPerSM=64)]
ARITH = dict(exact=abi.ARITH_EXACT, fma=abi.ARITH_FMA, dw=abi.ARITH_DW)


def _limit():
    import torch
    return 256 * torch.cuda.get_device_properties(0).multi_processor_count


def _spec(kind, law, arith, n=2500):
    kw = dict(law=law, arith=ARITH[arith])
    edge = 0.0135 * n ** (1.0 / 3.0)
    if kind == "peri":
        return scenes.periodic_cloud(n, 3, size=(edge,) * 3, dense=0.88, shear=0.3, **kw)
    # sparse: few spheres touch, and the spin of half of them is zero, so that warps hold any number of spinning ones
    spec = scenes.random_cloud(n, 3, box=(edge,) * 3, dense=0.99 if kind == "sparse" else 0.8, **kw)
    if kind == "sparse":
        still = np.random.default_rng(2).random(spec.particles.n) < np.linspace(0, 1, spec.particles.n)
        spec.particles.angVel[still] = 0
    return spec


@pytest.mark.parametrize("arith", ["exact", "fma", "dw"])
@pytest.mark.parametrize("kind, law", [("dense", "frict"), ("dense", "hertz"), ("sparse", "hertz"), ("peri", "frict"), ("peri", "hertz")])
def test_routes_agree(wdem_lib, kind, law, arith):
    spec = _spec(kind, law, arith)
    n = spec.particles.n
    a = gpu_handle(spec, keep_geom=False)
    others = [gpu_handle(spec, keep_geom=False) for _ in TWO_PASS]
    for h, shape in zip(others, TWO_PASS):
        h.set_launch_shape(**shape)
    for k in (1, 30, 50):
        a.step(k)
        pa, ca = gpu_particles(a, n), a.download_contacts()
        for h in others:
            h.step(k)
            assert_same_particles(gpu_particles(h, n), pa, ori_tol=0)
            assert_same_contacts(h.download_contacts(), ca)
    touched = len(np.unique(np.concatenate([ca.idA, ca.idB])[np.tile(ca.real == 1, 2)]))
    assert touched > n // 8 if kind == "dense" else touched > 0


def test_a_launch_shape_selects_the_two_passes(wdem_lib):
    """One launch a step more than the default shape's, in steps without a rebuild (a cloud that starts to fall)."""
    spec = scenes.random_cloud(500, 3, box=(0.12, 0.12, 0.12), vel_scale=0.0, angvel_scale=0.0)
    counts = []
    for shape in [None] + TWO_PASS:
        h = gpu_handle(spec)
        if shape:
            h.set_launch_shape(**shape)
        h.set_queue_depth(1)
        h.step(2)
        c = h.launch_count()
        h.step(3)
        counts.append(h.launch_count() - c)
        assert h.status().nFullRuns == 1
    assert counts[1:] == [counts[0] + 3] * 3


@pytest.mark.parametrize("more", [0, 1])
@pytest.mark.parametrize("kind", ["peri", "dense"])
def test_both_sides_of_the_limit_exact(wdem_lib, kind, more):
    """The largest scene of one launch and the smallest of two passes, against the oracle."""
    n = _limit() + more
    spec = _spec(kind, "frict", "exact", n if kind == "peri" else n - 6)
    assert spec.particles.n == n
    h = gpu_handle(spec, keep_geom=False)
    o = bridge.Oracle(spec.params, spec.particles, cell=spec.cell)
    for k in (1, 9):
        h.step(k)
        o.step(k)
        assert_same_particles(gpu_particles(h, n), o.particles())
    assert np.array_equal(np.sort(h.download_contacts().keys()), np.sort(o.contacts().keys()))


@pytest.mark.parametrize("more", [0, 1])
@pytest.mark.parametrize("law, arith", [("frict", "fma"), ("hertz", "fma"), ("hertz", "dw")])
def test_both_sides_of_the_limit_contracted(wdem_lib, law, arith, more):
    """The contracted variants on both sides: a step from a settled state, contact forces, particle forces and torques
    within 1e-12 of the largest of the exact variant's (each force's terms are rounded at their own size, some of
    them cancel), positions within 1e-15."""
    n = _limit() + more
    spec = _spec("dense", law, "exact", n - 6)
    assert spec.particles.n == n
    h = gpu_handle(spec, keep_geom=False)
    h.step(60)
    pa, ca, step = h.download_particles(spec.particles.copy()), h.download_contacts(), h.status().step
    h.close()
    he, hf = _handle(spec, pa, ca, step, abi.ARITH_EXACT), _handle(spec, pa, ca, step, ARITH[arith])
    he.step(1)
    hf.step(1)
    ce, cf = he.download_contacts(), hf.download_contacts()
    ce, cf = ce.take(ce.real == 1), cf.take(cf.real == 1)
    assert ce.n > 20000 and np.array_equal(ce.keys(), cf.keys())
    pe, pf = gpu_particles(he, n), gpu_particles(hf, n)
    for a, b in ((ce.force, cf.force), (pe.force, pf.force), (pe.torque, pf.torque)):
        assert np.abs(a - b).max() <= 1e-12 * np.abs(a).max()
    assert np.abs(pe.pos - pf.pos).max() <= 1e-15
