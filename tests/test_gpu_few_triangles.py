"""The exact path on both sides of the line under which the triangles are tried one by one (256
triangles, 2^23 pairs of voxel and triangle): distances and sides are the same."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T", [1, 5, 12, 255, 256, 257])
@pytest.mark.parametrize("dims", [(1, 1, 1), (5, 3, 4), (8, 8, 8), (9, 12, 20), (33, 31, 32), (32, 32, 33), (60, 61, 59),
                                  (89, 88, 90)])
def test_both_sides_of_the_line(engine, T, dims):
    from gbsdf import meshgen

    v, f = meshgen.perturbed_sphere(seed=3, n_lat=12, n_lon=24)
    s = 0.3 * max(dims)
    t = meshgen.to_triangles(np.asarray(v) * (s / 30.0) + (0.21, 0.13, 0.34), np.asarray(f)[-T:])
    mn = -(np.asarray(dims) // 2)
    mx = mn + np.asarray(dims) - 1
    a, ra = engine.compute_mesh_sdf(t, 1.0, mn, mx, path=engine.PATH_LEGACY, winding_eval=0)
    b, rb = engine.compute_mesh_sdf(t, 1.0, mn, mx, path=engine.PATH_LEGACY, winding_eval=1)
    assert ra.ok and rb.ok
    assert np.array_equal(np.signbit(a), np.signbit(b))
    assert np.abs(a - b).max() <= 2.0 ** -22 * max(dims)
    one_by_one = T <= 256 and T * int(np.prod(dims)) <= 1 << 23
    if one_by_one:
        assert np.array_equal(a.view(np.uint32), b.view(np.uint32)) and ra.stats["winding_certified"] == 0
