"""The parity pass at the edges of its work layout, both kinds of crossings, bit for bit against
the oracle: strips of 32 columns, supercell rows, tiles of 1,024 sign words, lists longer than
a CTA's step, triangles that a lane each takes (a fine mesh) and that the lanes take column by
column (a coarse one), and columns of more crossings than a column keeps."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _box(lo, hi):
    v = np.array([[x, y, z] for z in (lo[2], hi[2]) for y in (lo[1], hi[1]) for x in (lo[0], hi[0])], np.float64)
    f = np.array([[0, 2, 1], [1, 2, 3], [4, 5, 6], [5, 7, 6], [0, 1, 4], [1, 5, 4], [2, 6, 3], [3, 6, 7],
                  [0, 4, 2], [2, 4, 6], [1, 3, 5], [3, 7, 5]])
    return v, f


def _case(kind, dims, h=1.0):
    from gbsdf import meshgen

    ext = (np.asarray(dims) - 1) * h
    if kind == "fine":
        v, f = meshgen.perturbed_sphere(seed=4, n_lat=90, n_lon=180)
        v = np.asarray(v, np.float64)
        v = (v - v.min(0)) / (v.max(0) - v.min(0)) * (0.9 * ext) + 0.047 * ext
        parts = [(v, f)]
    elif kind == "coarse":
        parts = [_box(0.11 * ext, 0.83 * ext), _box(0.3 * ext, 0.95 * ext)]
    else:  # "slabs": more than 128 crossings in the columns through them
        zs = np.linspace(0.05, 0.9, 70) * ext[2]
        parts = [_box((0.1 * ext[0], 0.1 * ext[1], z), (0.6 * ext[0], 0.8 * ext[1], z + 0.004 * ext[2])) for z in zs]
    vs, fs, base = [], [], 0
    for v, f in parts:
        vs.append(v)
        fs.append(np.asarray(f) + base)
        base += len(v)
    v = np.concatenate(vs).astype(np.float32)
    tris = meshgen.to_triangles(v, np.concatenate(fs))
    return tris, np.zeros(3, np.int32), (np.asarray(dims) - 1).astype(np.int32), h


@pytest.mark.parametrize("dims", [(24, 24, 24), (31, 4, 40), (33, 30, 5), (64, 7, 33), (65, 61, 30), (12, 9, 1023),
                                  (9, 12, 1024), (34, 10, 1025), (8, 8, 2100)])
@pytest.mark.parametrize("kind", ["fine", "coarse", "slabs"])
@pytest.mark.parametrize("mode", ["REFERENCE", "EXACT_SIGNS"])
def test_parity_strips(engine, oracle, dims, kind, mode):
    tris, mn, mx, h = _case(kind, dims)
    exact = mode == "EXACT_SIGNS"
    st, ref, _, ost = oracle.fast_sdf(tris, h, mn, mx, fsm_mode=0, gwn_mode=1, signed_parity=exact)
    out, res = engine.compute_mesh_sdf(tris, h, mn, mx, mode=getattr(engine, "MODE_" + mode), path=engine.PATH_FAST,
                                       raise_on_error=False)
    assert res.ok == (st == oracle.OK)
    if not res.ok:  # declined by both
        return
    assert res.stats["unknown_columns"] == ost["unknown_columns"]
    if kind == "slabs" and min(dims[:2]) > 4:
        assert res.stats["unknown_columns"] > 0
    assert np.array_equal(out.view(np.uint32), ref.view(np.uint32))
