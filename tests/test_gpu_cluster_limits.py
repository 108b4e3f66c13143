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


@pytest.mark.parametrize("flat,whole", [(8, 8), (8, 1), (8, 40), (64, 8), (1, 8), (128, 2048), (24, 0)])
def test_nearest_cluster_without_area(engine, flat, whole):
    tris = _soup(np.random.default_rng(7), flat, whole)
    mn, mx = (0, 0, 0), (37, 38, 36)
    a, ra = engine.compute_mesh_sdf(tris, 1.0, mn, mx, path=engine.PATH_LEGACY, winding_eval=0)
    b, rb = engine.compute_mesh_sdf(tris, 1.0, mn, mx, path=engine.PATH_LEGACY, winding_eval=1)
    assert ra.ok and rb.ok
    assert np.array_equal(np.signbit(a), np.signbit(b))
    # the two minima may differ by the rounding of one squared distance
    assert np.abs(a - b).max() <= 2.0 ** -22 * 40.0
