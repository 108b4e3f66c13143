"""Iso-surface extraction at the edges of its work layout (words of 32 voxels, warps of 8 words,
blocks of 256 words) against the oracle, bit for bit: row lengths around the word and the
8-word chunk, lattices two voxels thick, full words (every cube cut), sparse crossings in one
word of a block, infinities and NaN, a seal lost to rounding, and outputs kept on the device."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _table():
    from gbsdf import _lib

    t = np.zeros((256, 16), np.int8)
    assert _lib.load().gbsdf_iso_surface_table(t.ctypes.data) == 0
    return t


@pytest.mark.parametrize("dims", [(2, 2, 2), (31, 2, 3), (32, 3, 2), (33, 9, 2), (34, 2, 9), (64, 5, 5), (65, 6, 4),
                                  (255, 3, 3), (257, 4, 5), (290, 7, 3), (32, 16, 17), (513, 5, 4)])
@pytest.mark.parametrize("kind", ["noise", "checker", "sparse", "nonfinite", "rounded_seal"])
def test_words_and_blocks(engine, oracle, dims, kind):
    import torch

    rng = np.random.default_rng(dims[0] * 100 + dims[1])
    g = rng.normal(0, 1, dims[::-1]).astype(np.float32)
    iso = np.float32(0.0)
    z, y, x = np.indices(g.shape)
    if kind == "checker":
        g = np.where((x + y + z) & 1, np.float32(0.5), np.float32(-0.25)).astype(np.float32)
    elif kind == "sparse":
        g = np.full(g.shape, 3.0, np.float32)
        g.reshape(-1)[rng.integers(0, g.size, 3)] = -1.0
    elif kind == "nonfinite":
        g[rng.random(g.shape) < 0.1] = np.inf
        g[rng.random(g.shape) < 0.1] = -np.inf
        g[rng.random(g.shape) < 0.1] = np.nan
    elif kind == "rounded_seal":  # iso + h rounds to iso: sealed voxels read as inside
        iso = np.float32(2.0 ** 24)
        g = (g * 8 + iso).astype(np.float32)
    args = (dims, 0.25, (-1.5, 2.0, 0.125), float(iso))
    v, i = engine.extract_iso_surface(g, *args)
    ov, oi = oracle.extract_iso_surface(g, *args, _table())
    assert np.array_equal(v.view(np.uint32), ov.view(np.uint32))
    assert np.array_equal(i, oi)
    dv, di = engine.extract_iso_surface(torch.from_numpy(g.copy()).cuda().ravel(), *args, outputs_on_device=True)
    assert np.array_equal(dv.cpu().numpy().view(np.uint32), ov.view(np.uint32))
    assert np.array_equal(di.cpu().numpy().view(np.uint32), oi)
