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


@pytest.mark.parametrize("n", [1017, 1018, 1019, 2042, 4500])
def test_rows_of_walls_at_range_edges(wdem_lib, n):
    """Bodies (with 6 walls) around multiples of 1024, where a wall's row gets another range of partner ids: the
    force sums need every row in the order of the partner ids, the carry finds old contacts in it."""
    side = 0.0125 * np.ceil(n ** (1.0 / 3.0))  # room for the generator to place all n
    spec = scenes.random_cloud(n, n, box=(side, side, side), rmin=0.004, rmax=0.005, dense=0.8)
    assert spec.particles.n == n + 6
    h, o = _run_both(spec, (1, 4, 40))
    assert h.status().nFullRuns == o.n_full_runs() > 1


@pytest.mark.parametrize("n", [1, 2, 4095, 4096, 4097, 12289, 135000])
def test_pairs_at_scan_tile_edges(wdem_lib, n):
    """Box pairs for counts at the edges of the scan's tiles (4096 values) and, last, beyond the 32 tiles that one
    look-back reads at a time; the pair set is known: boxes on a line, each meeting the next two."""
    k = np.random.default_rng(n).permutation(n)
    lo = np.stack([k * 1.0, np.zeros(n), np.zeros(n)], axis=1)
    h = abi.Handle(n)
    got = h.collide_boxes(lo, lo + np.array([2.5, 1.0, 1.0]), np.full(n, 5, np.uint32), 2)
    at = np.argsort(k)
    want = np.concatenate([np.stack([at[:-d], at[d:]], axis=1) for d in (1, 2) if n > d] + [np.zeros((0, 2), int)])
    want = np.sort(want, axis=1)
    assert np.array_equal(got, want[np.lexsort((want[:, 1], want[:, 0]))])


@pytest.mark.parametrize("size, n", [((0.03, 0.06, 0.045), 60), ((0.045, 0.045, 0.045), 70), ((0.1, 0.034, 0.034), 80),
                                     ((0.055, 0.04, 0.1), 150), ((0.1, 0.1, 0.1), 700)])
def test_periodic_grids_of_few_cells(wdem_lib, size, n):
    """Cells of the pair search from 1 to 8 per axis: with fewer than 3 along an axis both neighbours are the same
    cell and all neighbouring cells are searched by id, otherwise the cells ahead only."""
    spec = scenes.periodic_cloud(n, 5, size=size, shear=0.15)
    h, o = _run_both(spec, (1, 15))
    assert np.array_equal(h.download_contacts().cellDist, o.contacts().cellDist)


@pytest.mark.parametrize("periodic", [False, True])
def test_more_pairs_than_the_sweep_keeps(wdem_lib, periodic):
    """Large spheres among small ones: bodies with more partners than the counting walk keeps are walked again."""
    kw = dict(rmin=0.0012, rmax=0.009, dense=0.95, verletDist=0.0015)
    spec = scenes.periodic_cloud(900, 8, size=(0.07, 0.07, 0.07), **kw) if periodic else scenes.random_cloud(
        900, 8, box=(0.07, 0.07, 0.07), **kw)
    h, _ = _run_both(spec, (1, 20))
    c = h.download_contacts()
    assert np.bincount(np.concatenate([c.idA, c.idB])).max() > 40


@pytest.mark.parametrize("depth, graphs", [(2, abi.GRAPHS_OFF), (32, abi.GRAPHS_OFF), (32, abi.GRAPHS_ON)])
def test_energy_of_queued_steps(wdem_lib, depth, graphs):
    """Energy sums of queued steps, with collider rebuilds inside the queues, equal those of single steps bitwise."""
    spec = scenes.random_cloud(700, 6, dense=0.85, trackEnergy=1)
    a, b = gpu_handle(spec), gpu_handle(spec)
    a.set_queue_depth(1)
    b.set_queue_depth(depth)
    b.set_step_graphs(graphs)
    for k in (3, 60, 1, 130):
        a.step(k)
        b.step(k)
        assert a.energy() == b.energy()
    assert b.status().nFullRuns == a.status().nFullRuns > 3


@pytest.mark.parametrize("n", [2041, 2042, 2043, 4096])
def test_energy_sums_at_slice_edges(wdem_lib, n):
    """Particle counts (with 6 walls) around multiples of 2048, where the sums get another block: the energies agree
    with the oracle's, whose sums run in another order, to 1e-12."""
    side = 0.0125 * np.ceil(n ** (1.0 / 3.0))
    spec = scenes.random_cloud(n, n, box=(side, side, side), rmin=0.004, rmax=0.005, dense=0.8, trackEnergy=1)
    h = gpu_handle(spec)
    o = bridge.Oracle(spec.params, spec.particles)
    h.step(5)
    o.step(5)
    eg, eo = h.energy(), o.energy()
    eo = eo if isinstance(eo, dict) else dict(zip(abi.ENERGY_NAMES, eo))
    for k in abi.ENERGY_NAMES:
        assert abs(eg[k] - eo[k]) <= 1e-12 * max(abs(eo[k]), 1e-300), k


@pytest.mark.parametrize("n", [1, 31, 127, 128, 129, 700])
def test_network_gradient_at_tile_edges(wdem_lib, n):
    """Gradient and loss of the warm-start network for record counts around a tile of 128 (odd counts leave half of
    a sample pair's exchange to a padded sample), against the numpy restatement with the same BF16 rounding points.
    An FP32 sum in another order can move an activation across a BF16 rounding boundary, by 2^-8 of itself; with
    two such flips in the path of the largest entry a layer's gradients agree to 2^-7 of it, taken as 1e-2."""
    from oracle import warm_mlp
    rng = np.random.default_rng(n)
    w = warm_mlp.init(3).astype(np.float32)
    R = rng.uniform(-0.8, 0.8, (n, 17)).astype(np.float32)
    h = abi.Handle(1)
    h.warm_set_weights(w)
    g, loss = h.warm_grad(R)
    want_loss, want = warm_mlp.loss_grad(w, R.astype(np.float64))
    assert abs(loss - want_loss) <= 1e-2 * want_loss
    for (Wg, bg), (Wr, br) in zip(warm_mlp.unpack(g), warm_mlp.unpack(want)):
        assert np.abs(Wg - Wr).max() <= 1e-2 * np.abs(Wr).max()
        assert np.abs(bg - br).max() <= 1e-2 * np.abs(br).max()
