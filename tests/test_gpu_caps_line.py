"""Columns through holes decided by crossings and caps, and by the clusters alone below a number of
marked voxels (4,096 and one in 16,384 of the lattice): the sides are those of the triangle sum on
both sides of the line, in single builds and in patch rounds."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [48, 61, 96, 130])
@pytest.mark.parametrize("mode", ["EXACT_SIGNS", "REFERENCE"])
def test_marked_columns(engine, n, mode):
    from gbsdf import meshgen

    rng = np.random.default_rng(n)
    v, f = meshgen.perturbed_sphere(seed=2, n_lat=30, n_lon=60)
    f = np.asarray(f)
    marked = []
    for missing in (1, 8, 60, 200):
        vf, mn, mx = meshgen.fit_to_lattice(v, (n, n, n), 1.0, pad_voxels=3)
        tris = meshgen.to_triangles(vf, np.delete(f, rng.choice(len(f), missing, replace=False), 0))
        a, ra = engine.compute_mesh_sdf(tris, 1.0, mn, mx, mode=getattr(engine, "MODE_" + mode), path=engine.PATH_FAST,
                                        winding_eval=0, raise_on_error=False)
        b, rb = engine.compute_mesh_sdf(tris, 1.0, mn, mx, mode=getattr(engine, "MODE_" + mode), path=engine.PATH_FAST,
                                        winding_eval=1, raise_on_error=False)
        assert ra.status == rb.status
        if ra.ok:
            assert np.array_equal(a.view(np.uint32), b.view(np.uint32))
        assert ra.stats["fixup_voxels"] == rb.stats["fixup_voxels"]
        marked.append(ra.stats["fixup_voxels"] + ra.stats["patched_voxels"])
    assert max(marked) > 4096 + n ** 3 // 16384
