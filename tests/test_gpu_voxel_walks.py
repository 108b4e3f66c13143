"""Sides of marked voxels by walks, one voxel at a time, and by blocks of bricks (more than 2^18
marks and four for each triangle), for meshes that caps close and for those that keep to their own
clusters, against the triangle sum; rows that do not fill their last sign word."""
import numpy as np
import pytest
from test_gpu_clusters import KINDS, _compare, _mesh

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("dims,h", [((41, 39, 38), 0.7),       # walks
                                    ((73, 66, 70), 0.4),       # blocks of one brick
                                    ((145, 139, 141), 0.2)])   # of eight
def test_walks_and_blocks(engine, kind, dims, h):
    mn = -(np.asarray(dims) // 2)
    _compare(engine, _mesh(kind), h, mn, mn + np.asarray(dims) - 1)


def test_walks_of_dense_triangles(engine):
    # more than 2^18 marks, but fewer than four for each triangle
    from gbsdf import meshgen

    rng = np.random.default_rng(4)
    v, f = meshgen.perturbed_sphere(seed=1, n_lat=170, n_lon=340, base_radius=20.0)
    for missing in (0.0, 0.1):
        t = meshgen.to_triangles(np.asarray(v) + (0.31, 0.17, 0.23), np.asarray(f)[rng.random(len(f)) >= missing])
        assert 4 * len(t) > 66 * 65 * 70 > 1 << 18
        _compare(engine, t, 1.0, (-33, -32, -35), (32, 32, 34))


def test_marks_in_padded_rows(engine):
    # fast path, rows of 33 to 63 voxels: the sign words' pad bits are no voxels
    from gbsdf import meshgen

    rng = np.random.default_rng(6)
    v, f = meshgen.perturbed_sphere(seed=2, n_lat=30, n_lon=60)
    f = np.delete(np.asarray(f), rng.choice(len(f), 60, replace=False), 0)
    for n in (33, 47, 63):
        vf, mn, mx = meshgen.fit_to_lattice(v, (n, n, n), 1.0, pad_voxels=3)
        t = meshgen.to_triangles(vf, f)
        a, ra = engine.compute_mesh_sdf(t, 1.0, mn, mx, mode=engine.MODE_EXACT_SIGNS, path=engine.PATH_FAST)
        b, rb = engine.compute_mesh_sdf(t, 1.0, mn, mx, mode=engine.MODE_EXACT_SIGNS, path=engine.PATH_FAST, winding_eval=1)
        assert ra.stats["fixup_voxels"] == rb.stats["fixup_voxels"] > 0
        assert np.array_equal(a.view(np.uint32), b.view(np.uint32))
