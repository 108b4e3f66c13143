"""The orientation pass by union-find against a restatement of its rule (the label sweeps, in
numpy): random triangle numberings, many components, links that contradict each other (where
the sweeps decide the flips), and calls from several threads that share the kept scratch."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _sweeps(faces):
    """(flip per triangle, orientable, inconsistent) by the sweeps' rule."""
    T = len(faces)
    edges = {}
    for t, f in enumerate(faces):
        for e in range(3):
            u, v = int(f[e]), int(f[(e + 1) % 3])
            if u != v:
                edges.setdefault((min(u, v), max(u, v)), []).append((t, u < v))
    links = [[] for _ in range(T)]
    bad = False
    for uses in edges.values():
        if len(uses) == 2 and uses[0][0] != uses[1][0]:
            same = uses[0][1] == uses[1][1]
            bad |= same
            links[uses[0][0]].append((uses[1][0], same))
            links[uses[1][0]].append((uses[0][0], same))
    for k in links:
        k.sort()
    comp, flip = list(range(T)), [False] * T
    while True:
        nc, nf = list(comp), list(flip)
        for t in range(T):
            for n, same in links[t]:
                if comp[n] < nc[t]:
                    nc[t], nf[t] = comp[n], flip[n] ^ same
        if nc == comp and nf == flip:
            break
        comp, flip = nc, nf
    ok = all((flip[n] ^ same) == flip[t] for t in range(T) for n, same in links[t])
    return np.asarray(flip) & bad, ok, bad


def _sphere(n):
    from gbsdf import meshgen

    v, f = meshgen.perturbed_sphere(seed=n, n_lat=n, n_lon=2 * n)
    return np.asarray(v, np.float32), np.asarray(f, np.int64)


def _moebius(n, twist):
    a = np.arange(n)
    ang = 2 * np.pi * a / n
    w = ang / 2 * twist
    v = np.concatenate([np.stack([(3 + s * np.cos(w)) * np.cos(ang), (3 + s * np.cos(w)) * np.sin(ang), s * np.sin(w)], 1)
                        for s in (-1, 1)]).astype(np.float32)
    b, last = (a + 1) % n, a == n - 1
    lo, hi = np.where(last & (twist % 2 == 1), b + n, b), np.where(last & (twist % 2 == 1), b, b + n)
    return v, np.concatenate([np.stack([a, lo, a + n], 1), np.stack([a + n, lo, hi], 1)])


def _mesh(kind, seed):
    rng = np.random.default_rng(seed)
    parts = {"sphere": [_sphere(9)], "spheres": [_sphere(4 + k) for k in range(5)], "tiny": [_sphere(3)],
             "moebius": [_moebius(24, 1)], "mixed": [_sphere(6), _moebius(17, 1), _moebius(20, 2)]}[kind]
    vs, fs, base = [], [], 0
    for k, (v, f) in enumerate(parts):
        vs.append(v + np.float32(10 * k))
        fs.append(f + base)
        base += len(v)
    f = np.concatenate(fs)
    f = f[rng.permutation(len(f))]
    fl = rng.random(len(f)) < 0.4
    f[fl] = f[fl][:, [0, 2, 1]]
    f = np.concatenate([f, [[base, base, base + 1], [base, base + 1, base]]])  # degenerate: no link
    return np.concatenate(vs + [np.zeros((2, 3), np.float32)]), f.astype(np.uint32)


@pytest.mark.parametrize("kind", ["tiny", "sphere", "spheres", "moebius", "mixed"])
@pytest.mark.parametrize("seed", [0, 1, 2])
def test_unions_match_sweeps(engine, kind, seed):
    v, f = _mesh(kind, seed)
    flip, ok, bad = _sweeps(f)
    want = f.copy()
    want[flip] = want[flip][:, [0, 2, 1]]
    idx, orientable, inconsistent, inverted, vol = engine.orient_mesh(v, f)
    if inverted:
        want = want[:, [0, 2, 1]]
    assert (orientable, inconsistent) == (ok, bad)
    assert orientable == (kind not in ("moebius", "mixed"))
    assert np.array_equal(idx.reshape(-1, 3), want)


def test_kept_scratch_threads(engine):
    """Two sizes at once from four threads, and the scratch given back in between."""
    from gbsdf import _lib

    meshes = [_mesh("spheres", 3), _mesh("mixed", 4)]
    want = [engine.orient_mesh(v, f)[0] for v, f in meshes]
    bad = []

    def work(k):
        for r in range(20):
            v, f = meshes[(k + r) % 2]
            if not np.array_equal(engine.orient_mesh(v, f)[0], want[(k + r) % 2]):
                bad.append((k, r))
            if k == 0 and r == 10:
                _lib.load().gbsdf_release_workspace(0)

    threads = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad
