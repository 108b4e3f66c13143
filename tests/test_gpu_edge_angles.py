"""The triangle-by-triangle sum at voxels next to triangle edges, where both terms of the solid angle's
tangent cancel in FP32: long edges that pass a voxel at some ten-thousandths of a voxel, against the
winding number in FP64."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _winding(t, p):
    a, b, c = (t[:, k] - p for k in range(3))
    la, lb, lc = (np.linalg.norm(x, axis=1) for x in (a, b, c))
    det = np.einsum("ij,ij->i", a, np.cross(b, c))
    den = la * lb * lc + (a * b).sum(1) * lc + (b * c).sum(1) * la + (c * a).sum(1) * lb
    w = 2.0 * np.arctan2(det, den)
    w[(la <= 1e-6) | (lb <= 1e-6) | (lc <= 1e-6)] = 0.0  # the formula's rule at a vertex
    return w.sum() / (4.0 * np.pi)


def _soup(rng, n, side, length):
    """`n` triangles of up to `length` voxels, an edge of each 1e-5 to 1e-3 voxel beside a voxel; the voxels."""
    x = rng.integers(0, side, (n, 3)).astype(np.float64)
    u = rng.normal(size=(n, 3))
    u /= np.linalg.norm(u, axis=1)[:, None]
    q = np.cross(u, rng.normal(size=(n, 3)))
    q /= np.linalg.norm(q, axis=1)[:, None]
    e = x + q * 10.0 ** rng.uniform(-4.9, -3.0, (n, 1))
    s = length * rng.uniform(0.3, 1.0, (n, 2, 1))
    third = e + length * rng.uniform(0.3, 1.0, (n, 1)) * np.where(rng.random((n, 1)) < 0.7, -1, 1) * q
    third += 0.3 * length * rng.normal(size=(n, 3)) * rng.choice([0.0, 1e-4, 1.0], (n, 1))
    t = np.stack([e + u * s[:, 0], e - u * s[:, 1], third], 1)
    turn = rng.random(n) < 0.5
    t[turn] = t[turn][:, ::-1]
    return t.astype(np.float32), x.astype(int)


@pytest.mark.parametrize("winding_eval", [0, 1])
@pytest.mark.parametrize("length", [300.0, 1000.0])
def test_voxels_beside_long_edges(engine, length, winding_eval):
    checked = 0
    for seed in range(200):
        t, x = _soup(np.random.default_rng(seed), 24, 9, length)
        tris = np.concatenate([t.reshape(-1, 9), np.zeros((len(t), 3), np.float32)], 1)
        out, res = engine.compute_mesh_sdf(tris, 1.0, (0, 0, 0), (8, 8, 8), path=engine.PATH_LEGACY,
                                           winding_eval=winding_eval)
        assert res.ok
        for v in x:
            d = out[(v[2] * 9 + v[1]) * 9 + v[0]]
            w = abs(_winding(t.astype(np.float64), v.astype(np.float64)))
            if abs(d) > 1.1e-5 and abs(w - 0.5) > 1e-5:  # (nearer ones are on the surface: inside)
                assert np.signbit(d) == (w >= 0.5), (seed, v, d, w)
                checked += 1
    assert checked > 2000
