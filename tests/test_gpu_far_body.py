"""Bodies far from all others stretch the collider's grid until most bodies share one bucket of its sort: the pairs and
the run stay those of the oracle on both sides of the length where buckets are ranked no longer (2048), and the rebuild
does not cost the square of a bucket."""
import numpy as np
import pytest

from oracle import bridge
from woo_gb300 import abi, scenes

from helpers import assert_same_contacts, assert_same_particles, gpu_handle, gpu_particles

pytestmark = pytest.mark.gpu


def _lattice(n, r):
    s = int(np.ceil(n ** (1.0 / 3.0)))
    k = np.arange(n)
    c = np.stack([k % s, (k // s) % s, k // (s * s)], axis=1) + 0.5
    return (c + np.random.default_rng(n).uniform(-0.1, 0.1, (n, 3))) * 2.2 * r, s * 2.2 * r


def _pairs(lo, hi):
    """Overlapping pairs of boxes by sorting along x."""
    o = np.argsort(lo[:, 0], kind="stable")
    out = []
    end = np.searchsorted(lo[o, 0], hi[o, 0], side="right")
    for a in range(len(o)):
        i, j = o[a], o[a + 1:end[a]]
        ok = ((lo[i, 1:] <= hi[j, 1:]) & (hi[i, 1:] >= lo[j, 1:])).all(1)
        out.append(np.stack([np.full(ok.sum(), i), j[ok]], axis=1))
    p = np.sort(np.concatenate(out), axis=1)
    return p[np.lexsort((p[:, 1], p[:, 0]))]


@pytest.mark.parametrize("n", [2047, 2048, 2049, 2050, 4097, 4098, 6145, 8200, 20000])
@pytest.mark.parametrize("same", [False, True])
def test_pairs_with_a_body_far_away(wdem_lib, n, same):
    """n - 1 boxes together and one far away along every axis; same: the lower bounds along the sweep fall on a few
    values only, so that ties run over many bodies.  Buckets just below and above the limit, one tile of the sort to
    ten (odd counts too, with runs without a partner)."""
    c, edge = _lattice(n, 0.005)
    rng = np.random.default_rng(7)
    c = c[rng.permutation(n)]
    if same:
        c = np.round(c / 0.011) * 0.011
    c[n // 3] = 3e5 * edge
    h = abi.Handle(n)
    lo, hi = c - 0.0054, c + 0.0054
    got = h.collide_boxes(lo, hi, np.full(n, 5, np.uint32), 2)
    assert np.array_equal(got, _pairs(lo, hi))


@pytest.mark.parametrize("n", [1500, 3000])
def test_run_with_a_body_far_away(wdem_lib, n):
    """A squeezed cloud with one sphere far off, over several rebuilds: as the oracle, bit for bit."""
    spec = scenes.random_cloud(n, 3, box=(0.2, 0.2, 0.2), dense=0.85)
    assert spec.particles.n == n + 6
    spec.particles.pos[n // 2] += 4e4
    h = gpu_handle(spec)
    o = bridge.Oracle(spec.params, spec.particles)
    for k in (1, 4, 40):
        h.step(k)
        o.step(k)
        assert_same_particles(gpu_particles(h, n + 6), o.particles())
        assert_same_contacts(h.download_contacts(), o.contacts())
    assert h.status().nFullRuns == o.n_full_runs() > 2


def test_rebuild_time_with_a_body_far_away(wdem_lib):
    """1M spheres with one 10,000 edge lengths away along two axes, half of them in one bucket: 19 ms a rebuild (a
    radix sort took 20).  Each body ranked against its bucket took 149 ms."""
    n, r = 1000000, 0.005
    c, edge = _lattice(n, r)
    c[-1, :2] += 1e4 * edge
    mats = [dict(kind=abi.MAT_FRICT, density=2500.0, young=1e7, ktDivKn=0.2, tanPhi=0.5)]
    pa = scenes.assemble(c, np.full(n, r), 0, [], mats)
    ma = scenes.materials_array(mats)
    spec = scenes.SceneSpec(scenes.default_params(ma, dt=1e-7, verletDist=0.05 * r), ma, pa)
    h = gpu_handle(spec, keep_geom=False)
    h.set_timing(True)
    h.step(1)
    ms = []
    for _ in range(3):
        h.upload_particles(pa)
        h.step(1)
        ms.append(h.kernel_times()["collider"][0])
    assert min(ms) < 60.0, ms
