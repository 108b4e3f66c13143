"""The band splat by clusters against the oracle, and the exact path's cluster kernels (winding numbers by blocks of bricks, by crossings and caps,
nearest distances) against its per-triangle ones (winding_eval = 1) on every voxel: watertight,
holed, open, unwelded, degenerate and doubled meshes, ragged and tiny lattices, meshes partly
or wholly outside the lattice, both block sizes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _sphere(n=24, r=10.0, c=(0.3, 0.2, 0.1)):
    from gbsdf import meshgen

    v, f = meshgen.perturbed_sphere(seed=1, n_lat=n, n_lon=2 * n, base_radius=r, degree=3, coeff_scale=1.0)
    return np.asarray(v) + np.asarray(c), np.asarray(f)


def _mesh(kind):
    """(triangles, largest |coordinate|)"""
    from gbsdf import meshgen

    v, f = _sphere()
    rng = np.random.default_rng(5)
    if kind == "holes":  # single triangles and a larger patch missing
        keep = rng.random(len(f)) > 0.03
        keep[100:160] = False
        f = f[keep]
    elif kind == "open":  # an open shell: half of the surface
        f = f[: len(f) // 2]
    elif kind == "unwelded":  # every triangle its own vertices, moved a little
        v = v[f].reshape(-1, 3) + rng.normal(0.0, 1e-3, (3 * len(f), 3))
        f = np.arange(len(v)).reshape(-1, 3)
    elif kind == "doubled":  # a second, overlapping shell, one of the same orientation and one inside out
        w, g = _sphere(12, 6.0, (4.0, 0.0, 0.0))
        u, k = _sphere(10, 3.0, (-2.0, 0.0, 0.0))
        f = np.vstack([f, g + len(v), k[:, ::-1] + len(v) + len(w)])
        v = np.vstack([v, w, u])
    elif kind == "repeated":  # some triangles twice, some with both orientations
        f = np.vstack([f, f[:40], f[60:90, ::-1]])
    elif kind == "few":  # a box of twelve large triangles
        c = np.array([[x, y, z] for x in (-7.3, 8.1) for y in (-6.2, 9.4) for z in (-8.7, 7.9)])
        v = c
        q = [(0, 1, 3, 2), (4, 6, 7, 5), (0, 4, 5, 1), (2, 3, 7, 6), (0, 2, 6, 4), (1, 5, 7, 3)]
        f = np.array([t for a, b, c_, d in q for t in ((a, b, c_), (a, c_, d))])
    t = meshgen.to_triangles(v, f)
    if kind == "degenerate":  # points, needles and collinear triangles among the others
        e = t[:30].copy()
        e[:10, 3:9] = np.tile(e[:10, :3], 2)
        e[10:20, 6:9] = e[10:20, 3:6]
        e[20:, 6:9] = 0.5 * (e[20:, :3] + e[20:, 3:6])
        t = np.vstack([t, e]).astype(np.float32)
    return t


def _compare(engine, tris, h, mn, mx):
    a, ra = engine.compute_mesh_sdf(tris, h, mn, mx, path=engine.PATH_LEGACY, winding_eval=0)
    b, rb = engine.compute_mesh_sdf(tris, h, mn, mx, path=engine.PATH_LEGACY, winding_eval=1)
    assert ra.ok and rb.ok
    # a voxel on the surface is inside by its distance in both; elsewhere the sides are exact
    assert np.array_equal(np.signbit(a), np.signbit(b))
    # the per-triangle kernel skips a tile whose box is not below its best: the two minima may
    # differ by the rounding of one squared distance (coordinates of up to |c|, 2^-22 of them)
    c = max(np.abs(tris[:, :9]).max(), np.abs(np.asarray([mn, mx])).max() * h)
    assert np.abs(a - b).max() <= 2.0 ** -22 * c


KINDS = ["closed", "holes", "open", "unwelded", "doubled", "repeated", "few", "degenerate"]


@pytest.mark.parametrize("kind", KINDS)
def test_bricks(engine, kind):
    # 33 x 31 x 29 and more than 32,768 voxels (from which crossings and caps are used)
    tris = _mesh(kind)
    _compare(engine, tris, 0.9, (-18, -17, -16), (18, 17, 16))
    _compare(engine, tris, 0.9, (-16, -15, -14), (16, 15, 14))


@pytest.mark.parametrize("kind", ["holes", "doubled", "few"])
def test_blocks_of_bricks(engine, kind):
    # from 152 x 4 blocks of 16^3 the bricks are taken eight at a time; ragged sides
    _compare(engine, _mesh(kind), 0.2, (-70, -69, -65), (73, 72, 71))


@pytest.mark.parametrize("lattice", [((0, 0, 0), (0, 0, 0)), ((-3, 0, -2), (5, 0, 6)), ((-40, -2, -2), (40, 1, 0)),
                                     ((-8, -8, -40), (0, 0, 40)), ((30, 30, 30), (71, 66, 63)),
                                     ((-1000, -20, 900), (-960, 20, 935))])
def test_lattices(engine, lattice):
    # tiny, flat and long lattices; lattices beside and far from the mesh
    for kind in ("closed", "holes"):
        _compare(engine, _mesh(kind), 0.7, *lattice)


@pytest.mark.parametrize("n", [1, 7, 8, 9, 127, 128, 129, 2047, 2049])
def test_triangle_counts(engine, n):
    # the edges of the clusters' runs (8, 128 and 2048 triangles) and of the sort's tiles
    tris = _mesh("closed")[:n]
    _compare(engine, tris, 1.1, (-14, -13, -12), (15, 14, 13))


@pytest.mark.parametrize("kind,h,half", [(k, 0.9, (18, 17, 16)) for k in KINDS] +
                         [("few", 0.16, (66, 69, 64)),      # a cluster's box over more than 2048 bricks
                          ("closed", 4.0, (3, 4, 5)),       # hundreds of clusters in a brick
                          ("closed", 0.05, (20, 20, 20))])  # triangles larger than a brick
def test_band_splat(engine, oracle, kind, h, half):
    tris = _mesh(kind)
    mn, mx = -np.asarray(half), np.asarray(half) + (1, 0, 2)
    if kind == "closed" and h < 0.1:
        mn, mx = mn + (200, 0, 0), mx + (200, 0, 0)  # a window around the surface
    out, res = engine.compute_mesh_sdf(tris, h, mn, mx, mode=engine.MODE_EXACT_SIGNS, path=engine.PATH_FAST,
                                       raise_on_error=False)
    st, ref, _, ost = oracle.fast_sdf(tris, h, mn, mx, fsm_mode=0, gwn_mode=1, signed_parity=True)
    assert res.status == st and res.stats["band_voxels"] == ost["band_voxels"] > 0
    if st == oracle.OK:
        assert np.array_equal(out.view(np.uint32), ref.view(np.uint32))
