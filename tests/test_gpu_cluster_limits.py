"""Nearest distances where the cluster next to an octant has no area: the distance to a triangle
of two equal corners is not a number, the octant then has no limit, and it keeps every listed
cluster and nothing else."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _soup(rng, flat, whole):
    """`flat` triangles (a, a, c) in a clump below the lattice's corner, their third corners towards
    +x +y +z, so that none has a distance to any point of the lattice, and `whole` ordinary ones
    in another clump (clusters are runs of eight in Hilbert order)."""
    a = rng.uniform(-3.0, -1.0, (flat, 3))
    e = np.concatenate([a, a, a + rng.uniform(0.3, 0.9, (flat, 3))], 1)
    b = rng.uniform(26.0, 29.0, (whole, 1, 3)) + rng.uniform(-1.0, 1.0, (whole, 3, 3))
    t = np.concatenate([e, b.reshape(whole, 9)])
    return np.concatenate([t, np.zeros((flat + whole, 3))], 1).astype(np.float32)


@pytest.mark.parametrize("flat,whole", [(8, 256), (8, 249), (8, 4000), (64, 200), (1, 256), (128, 2048), (264, 0)])
def test_nearest_cluster_without_area(engine, flat, whole):
    tris = _soup(np.random.default_rng(7), flat, whole)
    mn, mx = (0, 0, 0), (37, 38, 36)
    a, ra = engine.compute_mesh_sdf(tris, 1.0, mn, mx, path=engine.PATH_LEGACY, winding_eval=0)
    b, rb = engine.compute_mesh_sdf(tris, 1.0, mn, mx, path=engine.PATH_LEGACY, winding_eval=1)
    assert ra.ok and rb.ok
    assert np.array_equal(np.signbit(a), np.signbit(b))
    # the two minima may differ by the rounding of one squared distance
    assert np.abs(a - b).max() <= 2.0 ** -22 * 40.0


def _mixed(rng, n, reach):
    """Clumps of triangles (a, a, c), whose distance exists on one side of them only, of ordinary
    triangles within `reach` of the lattice's middle part, and one of many at its far corner."""
    a = np.repeat(rng.uniform(8.0, 28.0, (n, 3)), 16, 0) + rng.uniform(-0.7, 0.7, (16 * n, 3))
    e = np.concatenate([a, a, a + rng.uniform(-0.9, 0.9, (16 * n, 3))], 1)
    c = np.repeat(rng.uniform(8.0, 28.0, (n, 3)), 8, 0)
    b = (c + rng.uniform(-reach, reach, (8 * n, 3)))[:, None] + rng.uniform(-1.0, 1.0, (8 * n, 3, 3))
    far = rng.uniform(33.0, 36.0, (256, 1, 3)) + rng.uniform(-0.3, 0.3, (256, 3, 3))  # so many that clusters are used
    t = np.concatenate([e, b.reshape(-1, 9), far.reshape(-1, 9)])
    return np.concatenate([t, np.zeros((len(t), 3))], 1).astype(np.float32)


@pytest.mark.parametrize("n,reach", [(1, 0.0), (1, 6.0), (3, 6.0), (20, 3.0), (200, 2.0)])
def test_limits_that_do_not_hold(engine, n, reach):
    # a centre on the side where such a triangle has a distance, voxels on the other: each voxel
    # still gets the least distance over every triangle
    for seed in range(4):
        tris = _mixed(np.random.default_rng(seed), n, reach)
        mn, mx = (0, 0, 0), (37, 38, 36)
        a, ra = engine.compute_mesh_sdf(tris, 1.0, mn, mx, path=engine.PATH_LEGACY, winding_eval=0)
        b, rb = engine.compute_mesh_sdf(tris, 1.0, mn, mx, path=engine.PATH_LEGACY, winding_eval=1)
        assert ra.ok and rb.ok
        assert np.abs(np.abs(a) - np.abs(b)).max() <= 2.0 ** -22 * 40.0


@pytest.mark.parametrize("n,reach", [(1, 0.0), (1, 6.0), (3, 6.0), (20, 3.0), (200, 2.0)])
def test_band_limits_that_do_not_hold(engine, oracle, n, reach):
    # the same in the band splat (8 voxels), against the oracle's
    for seed in range(3):
        tris = _mixed(np.random.default_rng(seed), n, reach)
        mn, mx = (0, 0, 0), (37, 38, 36)
        out, res = engine.compute_mesh_sdf(tris, 1.0, mn, mx, mode=engine.MODE_EXACT_SIGNS, path=engine.PATH_FAST,
                                           raise_on_error=False)
        st, ref, _, ost = oracle.fast_sdf(tris, 1.0, mn, mx, fsm_mode=0, gwn_mode=1, signed_parity=True)
        assert res.status == st and res.stats["band_voxels"] == ost["band_voxels"] > 0
        if st == oracle.OK:
            assert np.array_equal(np.abs(out).view(np.uint32), np.abs(ref).view(np.uint32))
