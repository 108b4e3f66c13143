"""Sides from crossings and caps against the triangle-by-triangle sum (winding_eval = 1), where the
heights of crossings are hard: windows on faces some ten thousand voxels across that run almost
along a lattice plane, slivers far from the origin, surfaces and caps through lattice points."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

QUADS = [(0, 1, 3, 2), (4, 6, 7, 5), (0, 4, 5, 1), (2, 3, 7, 6), (0, 2, 6, 4), (1, 5, 7, 3)]


def _tris(v, f):
    t = np.asarray(v, np.float64)[np.asarray(f)].reshape(-1, 9)
    return np.concatenate([t, np.zeros((len(t), 3))], 1).astype(np.float32)


def _split(v, f, k):
    """Each triangle of (v, f) in k^2 ones."""
    t = np.asarray(v, np.float64)[np.asarray(f)]
    p = lambda i, j: (t[:, 0] * (k - i - j) + t[:, 1] * i + t[:, 2] * j) / k
    out = [np.stack([p(i, j), p(i + 1, j), p(i, j + 1)], 1) for i in range(k) for j in range(k - i)]
    out += [np.stack([p(i + 1, j), p(i + 1, j + 1), p(i, j + 1)], 1) for i in range(k - 1) for j in range(k - 1 - i)]
    return np.concatenate(out).reshape(-1, 3), np.arange(3 * len(t) * k * k).reshape(-1, 3)


def _box(lo, hi, faces=range(6)):
    v = np.array([[x, y, z] for x in (lo[0], hi[0]) for y in (lo[1], hi[1]) for z in (lo[2], hi[2])], np.float64)
    return v, [t for q in faces for t in ((QUADS[q][0], QUADS[q][1], QUADS[q][2]),
                                          (QUADS[q][0], QUADS[q][2], QUADS[q][3]))]


def _compare(engine, tris, h, mn, mx):
    a, ra = engine.compute_mesh_sdf(tris, h, mn, mx, path=engine.PATH_LEGACY, winding_eval=0)
    b, rb = engine.compute_mesh_sdf(tris, h, mn, mx, path=engine.PATH_LEGACY, winding_eval=1)
    assert ra.ok and rb.ok
    wrong = np.flatnonzero(np.signbit(a) != np.signbit(b))
    assert len(wrong) == 0, (len(wrong), np.abs(b[wrong]).max() / h)
    inside = np.signbit(b).mean()
    assert 0.01 < inside < 0.99


@pytest.mark.parametrize("side", [300.0, 2000.0, 8000.0, 40000.0, 200000.0])
def test_window_on_a_large_face(engine, side):
    rng = np.random.default_rng(int(side))
    for k in range(6):
        # a face whose distance to the lattice's middle plane stays within some hundredths of a voxel
        slope = rng.uniform(-2e-4, 2e-4, 2)
        v, f = _box((-0.41 * side, -0.55 * side, -0.6 * side), (0.59 * side, 0.47 * side, 0.0))
        v[:, 2] += v[:, :2] @ slope + rng.uniform(-0.01, 0.01)
        axes = [(0, 1, 2), (1, 2, 0), (2, 0, 1)][k % 3]
        v = v[:, np.argsort(axes)]
        n = np.array([183, 182, 24])[np.argsort(axes)]  # (large enough that clusters and crossings are used)
        _compare(engine, _tris(v, f), 1.0, -n // 2, -n // 2 + n)


@pytest.mark.parametrize("at", [(0, 0, 0), (900, -700, 1100), (5000, 4000, -3000)])
@pytest.mark.parametrize("segments", [90, 720])
def test_slivers(engine, at, segments):
    # a tilted cylinder with its side in triangles of its whole length
    a = np.linspace(0.0, 2.0 * np.pi, segments, endpoint=False)
    ring = np.stack([14.0 * np.cos(a), 14.0 * np.sin(a)], 1)
    v = np.concatenate([np.column_stack([ring, np.full(segments, z)]) for z in (-150.0, 150.0)] + [[[0, 0, -150.0]],
                                                                                             [[0, 0, 150.0]]])
    i, j = np.arange(segments), (np.arange(segments) + 1) % segments
    f = np.concatenate([np.stack([i, j, j + segments], 1), np.stack([i, j + segments, i + segments], 1),
                        np.stack([j, i, np.full(segments, 2 * segments)], 1),
                        np.stack([i + segments, j + segments, np.full(segments, 2 * segments + 1)], 1)])
    for tilt in (0.7, 1.2, 1.56):
        c, s = np.cos(tilt), np.sin(tilt)
        r = np.array([[c, 0.0, s], [0.0, 1.0, 0.0], [-s, 0.0, c]]) @ np.array([[0.8, -0.6, 0.0], [0.6, 0.8, 0.0], [0, 0, 1.0]])
        tris = _tris(v @ r.T + np.asarray(at) + (0.13, 0.21, 0.34), f)
        mn = np.asarray(at) - 20
        _compare(engine, tris, 1.0, mn, mn + (41, 40, 42))


@pytest.mark.parametrize("faces", [range(6), [0, 1, 2, 3, 4], [0, 1, 3, 4, 5], [1, 2, 4]])
def test_surfaces_and_caps_through_lattice_points(engine, faces):
    mn, mx = (-20, -19, -18), (20, 21, 19)
    v, f = _split(*_box((-8, -8, -8), (8, 8, 8), faces), 8)
    _compare(engine, _tris(v, f), 1.0, mn, mx)
    # turned so that oblique faces, edges and vertices still meet lattice points
    r = np.array([[1, -1, 0], [1, 1, 0], [0, 0, 1]], np.float64)
    _compare(engine, _tris(v @ r.T, f), 1.0, mn, mx)
    _compare(engine, _tris(v @ (r @ np.array([[1, 0, 0], [0, 1, -1], [0, 1, 1]], np.float64)).T * 0.5, f), 1.0, mn, mx)


def test_octahedron_on_the_lattice(engine):
    v = 12.0 * np.array([[1, 0, 0], [-1, 0, 0], [0, 1, 0], [0, -1, 0], [0, 0, 1], [0, 0, -1]])
    f = np.array([(0, 2, 4), (2, 1, 4), (1, 3, 4), (3, 0, 4), (2, 0, 5), (1, 2, 5), (3, 1, 5), (0, 3, 5)])
    for keep in (slice(None), slice(1, None), slice(2, None)):
        _compare(engine, _tris(*_split(v, f[keep], 12)), 1.0, (-18, -17, -16), (18, 17, 16))
