"""A triangle's dipole about its FP32 centroid: with triangles of a few units in the last place, all
centroids rounded the same way, the rounding moves a patch's winding number by more than the
expansion's own rest. A voxel whose |w| is next to 1/2 must still get the side of the FP64 sum."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

V = np.array([20000.0, 20000.0, 20000.0])  # the voxel, at a voxel size of 1
ULP = 2.0 ** -9                             # of coordinates in 16384 .. 32768


def _winding(t, p):
    a, b, c = (t[:, k] - p for k in range(3))
    la, lb, lc = (np.linalg.norm(x, axis=1) for x in (a, b, c))
    det = np.einsum("ij,ij->i", a, np.cross(b, c))
    den = la * lb * lc + (a * b).sum(1) * lc + (b * c).sum(1) * la + (c * a).sum(1) * lb
    return np.arctan2(det, den).sum() / (2.0 * np.pi)


def _patch(up):
    """Triangles of 4 units in the last place, their third corner one unit higher, 0.31 below the
    voxel; their FP32 centroids lie a third of a unit lower than the true ones."""
    n = 154
    i, j = (x.ravel() * 4.0 * ULP for x in np.meshgrid(np.arange(-n // 2, n // 2), np.arange(-n // 2, n // 2)))
    z = np.full_like(i, -160.0 * ULP)
    L = 4.0 * ULP
    q = lambda x, y, w: np.stack([i + x, j + y, z + w], 1)
    t = np.concatenate([np.stack([q(0, 0, 0), q(L, 0, 0), q(L, L, up * ULP)], 1),
                        np.stack([q(0, 0, 0), q(L, L, up * ULP), q(0, L, 0)], 1)])
    return t + V


@pytest.mark.parametrize("up", [1.0, -1.0])
def test_sides_next_to_one_half(engine, up):
    patch = _patch(up)
    assert np.array_equal(patch, patch.astype(np.float32))
    w = _winding(patch, V)
    rng = np.random.default_rng(3)
    found = 0
    for _ in range(400):  # a triangle above the voxel that brings |w| next to 1/2
        a, z = 2.0 * np.pi * (np.arange(3) / 3.0 + rng.random()), rng.uniform(0.4, 0.9)
        ring = np.stack([np.cos(a), np.sin(a), np.zeros(3)], 1)
        if _winding(ring[None] + (0.0, 0.0, z), np.zeros(3)) * w < 0:
            ring = ring[::-1]
        lo, hi = 0.1, 20.0
        for _ in range(40):
            r = 0.5 * (lo + hi)
            lo, hi = (r, hi) if abs(w + _winding(r * ring[None] + (0.0, 0.0, z), np.zeros(3))) < 0.5 else (lo, r)
        lid = (r * ring + (0.0, 0.0, z) + V).astype(np.float32).astype(np.float64)
        off = abs(w + _winding(lid[None], V)) - 0.5
        if not 2e-5 < up * off < 2e-4:  # on the side that the rounding leads away from
            continue
        t = np.concatenate([patch, lid[None]]).reshape(-1, 9)
        tris = np.concatenate([t, np.zeros((len(t), 3))], 1).astype(np.float32)
        mn = V.astype(np.int32) - 2
        a0, ra = engine.compute_mesh_sdf(tris, 1.0, mn, mn + 4, path=engine.PATH_LEGACY, winding_eval=0)
        assert ra.ok
        assert np.signbit(a0[2 * 25 + 2 * 5 + 2]) == (off >= 0.0), off
        found += 1
        if found == 12:
            break
    assert found >= 6
