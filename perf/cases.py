"""The engine's work, as its users have it do it, in measurable cases.

A case goes through the public entry points of the package (``gbsdf``): mesh-to-SDF builds in
every mode and on both paths, a planned batch, the iso-surface of a device grid, the mesh
decoders and one training step of the sign-risk network. Sizes are those of the repository's
configurations and tests, or lie between them. ``listed()`` says for each case what it stands
for; ``draw()`` gives more of the same ranges.

A seed turns the mesh about the vertical axis and moves it by a fraction of a voxel (or,
where the lattice or the mesh must keep its size, draws noise on its vertices or values), so
that every input value changes with it.
"""
import functools
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.getcwd(), "rhizome_v24.15_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)
import gbsdf  # noqa: E402
from gbsdf import learn, meshgen  # noqa: E402

MODES = {"reference": gbsdf.MODE_REFERENCE, "exact_signs": gbsdf.MODE_EXACT_SIGNS, "exact": gbsdf.MODE_EXACT,
         "learned": gbsdf.MODE_LEARNED}
PATHS = {"auto": gbsdf.PATH_AUTO, "fast": gbsdf.PATH_FAST}


def listed():
    return [
        # The smallest builds: a preview-sized grid through the default dispatch (the exact
        # per-voxel path below 32M voxels), host arrays in and out. Latency and launches.
        dict(name="auto_mug_48", kind="sdf", mesh="mug", tris=2712, nx=48, ny=48, nz=52, h=1.6, mode="reference",
             path="auto", memory="host"),
        # The 128^3 mug at 0.8 mm on the fast path with the reference's signs and probes: an
        # ordinary interactive build (upright where its probes accept it).
        dict(name="fast_mug_128", kind="sdf", mesh="mug", tris=24000, nx=128, ny=128, nz=128, h=0.8,
             mode="reference", path="fast", memory="device"),
        # The application's mesh front-end at a coarse voxel size: indexed mesh on the host,
        # lattice from the mesh, default dispatch, host grid back.
        dict(name="auto_build_mug", kind="build", mesh="mug", tris=24000, nx=181, ny=141, nz=171, h=0.6),
        # A call just above the 32M-voxel dispatch line, odd sides, page-locked host arrays in
        # and out: the application's fast path at a middling voxel size.
        dict(name="auto_mug_333", kind="sdf", mesh="mug", tris=60000, nx=333, ny=331, nz=347, h=0.25,
             mode="exact_signs", path="auto", memory="pinned"),
        # The 0.10 mm mug, 650.8M voxels, signs by the winding number: the largest grid.
        dict(name="signs_mug_860", kind="sdf", mesh="mug", tris=179840, nx=860, ny=860, nz=880, h=0.1,
             mode="exact_signs", path="fast", memory="device"),
        # The defective vessel tree (holes, jitter, duplicated vertices) with the sign-risk
        # network's proposals.
        dict(name="learned_vessel_512", kind="sdf", mesh="vessel", tris=412455, nx=512, ny=512, nz=512, h=0.15,
             mode="learned", path="fast", memory="device"),
        # A noisy scanned surface with 1% of its triangles missing: many columns through holes
        # are decided by the winding number.
        dict(name="signs_blob_640", kind="sdf", mesh="blob", tris=800000, nx=640, ny=640, nz=640, h=0.16,
             mode="exact_signs", path="fast", memory="device"),
        # The converged, monotone distance update on a lattice with ragged sides.
        dict(name="exact_sphere_150", kind="sdf", mesh="sphere", tris=30000, nx=150, ny=143, nz=161, h=0.5,
             mode="exact", path="fast", memory="device"),
        # A scene of meshes of uneven size as one planned batch, replayed.
        dict(name="batch_16", kind="batch", n=16, layout=4, t_lo=2000, t_hi=150000, g_lo=64, g_hi=224,
             mode="exact_signs"),
        # Marching cubes of a grid on the device, the mesh left there.
        dict(name="iso_509", kind="iso", nx=509, ny=480, nz=512, h=0.2),
        # Opening a mesh file: decode, weld and orient a binary STL.
        dict(name="stl_180k", kind="file", format="stl", mesh="mug", tris=179840),
        # One step of training the sign-risk network: gradients, update, scores.
        dict(name="train_4096", kind="train", rows=4096),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["fast", "fast", "auto", "signs", "holes", "exact", "learned", "batch", "iso", "file", "train"])

    def sides(lo, hi):
        g = _log(rng, lo, hi)
        return dict(zip(("nx", "ny", "nz"), (max(24, g + rng.randint(-g // 12, g // 12)) for _ in range(3))))

    if kind == "fast":  # triangles as dense on the lattice as in the named mugs
        s = sides(56, 480)
        return dict(kind="sdf", mesh="mug", tris=min(150000, round(s["nx"] ** 2 * rng.uniform(0.25, 1.4))), **s,
                    h=rng.choice([0.1, 0.25, 0.5, 0.8]), mode="exact_signs", path="fast",
                    memory=rng.choice(["device", "pinned", "host"]))
    if kind == "auto":
        s = dict(mesh=rng.choice(["mug", "sphere"]), tris=_log(rng, 1500, 24000), **sides(36, 150),
                 h=rng.choice([0.5, 0.6, 0.8, 1.6]))
        if rng.random() < 0.5:
            return dict(kind="build", **s)
        return dict(kind="sdf", mode="reference", path="auto", memory="host", **s)
    if kind == "signs":
        return dict(kind="sdf", mesh="mug", tris=_log(rng, 8000, 179840), **sides(100, 640),
                    h=rng.choice([0.1, 0.15, 0.3]), mode="exact_signs", path="fast", memory="device")
    if kind == "holes":
        return dict(kind="sdf", mesh=rng.choice(["blob", "vessel"]), tris=_log(rng, 20000, 600000),
                    **sides(128, 512), h=rng.choice([0.15, 0.16, 0.3]), mode="exact_signs", path="fast",
                    memory="device")
    if kind == "exact":
        return dict(kind="sdf", mesh=rng.choice(["mug", "sphere"]), tris=_log(rng, 4000, 40000), **sides(72, 200),
                    h=rng.choice([0.3, 0.5, 0.8]), mode="exact", path="fast", memory="device")
    if kind == "learned":
        return dict(kind="sdf", mesh="vessel", tris=_log(rng, 20000, 200000), **sides(96, 320),
                    h=rng.choice([0.15, 0.3]), mode="learned", path="fast", memory="device")
    if kind == "batch":
        return dict(kind="batch", n=rng.randint(4, 16), layout=rng.randint(1, 1 << 20), t_lo=2000,
                    t_hi=_log(rng, 20000, 150000), g_lo=64, g_hi=rng.randint(96, 224), mode="exact_signs")
    if kind == "iso":
        return dict(kind="iso", **sides(96, 560), h=rng.choice([0.1, 0.2, 0.5]))
    if kind == "file":
        return dict(kind="file", format=rng.choice(["stl", "ascii_stl", "obj"]),
                    mesh=rng.choice(["mug", "sphere"]), tris=_log(rng, 3000, 120000))
    return dict(kind="train", rows=_log(rng, 512, 16384) | 1)


# ---- inputs ------------------------------------------------------------------------------
@functools.lru_cache(maxsize=64)
def _shape(mesh, tris):
    """(vertices FP64, faces) of about `tris` triangles."""
    if mesh == "mug":
        f = math.sqrt(tris / 23300.0)
        if tris == 179840:
            return meshgen.mug(segments=768, n_bottom=16, n_wall=37, n_rim=4, handle_path=96, handle_around=64)
        return meshgen.mug(segments=max(16, round(256 * f)), n_bottom=max(1, round(6 * f)), n_wall=max(2, round(14 * f)),
                           n_rim=max(1, round(2 * f)), handle_path=max(8, round(28 * f)),
                           handle_around=max(8, round(32 * f)))
    if mesh == "sphere":
        n = max(8, round(math.sqrt(tris / 4.0)))
        return meshgen.perturbed_sphere(seed=4, n_lat=n, n_lon=2 * n)
    if mesh == "vessel":
        if tris > 400000:
            return meshgen.vessel_tree(seed=3)
        levels = int(np.clip(round(math.log2(tris / 6000.0)), 2, 5))
        k = math.sqrt(tris / (2 ** (levels + 1) - 1) / 40.0)
        return meshgen.vessel_tree(seed=3, levels=levels, around=max(8, round(4 * k)), n_len=max(2, round(3 * k)),
                                   n_cap=max(1, round(k)))
    n = max(16, round(math.sqrt(tris / 4.0)))
    return meshgen.sh_blob(seed=5, n_lat=n, n_lon=2 * n)


@functools.lru_cache(maxsize=16)
def _shape_on_gpu(mesh, tris):
    v, f = _shape(mesh, tris)
    return torch.from_numpy(np.asarray(v, np.float64)).cuda(), torch.from_numpy(np.asarray(f, np.int64)).cuda()


def _place(v, dims, h, seed, span=None):
    """Vertices turned about z by the seed's angle and scaled and centred into the lattice
    (10 voxels free on the tightest axis, or the share `span` of the smallest side)."""
    r = np.random.RandomState(seed % (1 << 31))
    a = r.uniform(0.0, 2.0 * math.pi)
    off = r.uniform(0.0, 1.0, 3)
    rot = torch.tensor([[math.cos(a), -math.sin(a), 0.0], [math.sin(a), math.cos(a), 0.0], [0.0, 0.0, 1.0]],
                       dtype=torch.float64, device=v.device)
    v = v @ rot.T
    lo, hi = v.min(0).values, v.max(0).values
    ext = (hi - lo).cpu().numpy()
    d = np.asarray(dims)
    s = float(np.min((d - 1 - 20) * h / ext)) if span is None else float(span * (d.min() - 1) * h / ext.max())
    mn = -(d // 2)
    centre = torch.from_numpy((mn + (d - 1) / 2.0) * h + off * h).to(v.device)
    return ((v - (lo + hi) / 2.0) * s + centre).float(), mn.astype(np.int32), (mn + d - 1).astype(np.int32)


def _soup(v, f):
    """(T, 12) triangle records (v0, v1, v2, unit normal), degenerate faces dropped."""
    a, b, c = v[f[:, 0]], v[f[:, 1]], v[f[:, 2]]
    n = torch.linalg.cross(b - a, c - a)
    l2 = (n * n).sum(1)
    keep = l2 > 1e-12
    return torch.cat([a[keep], b[keep], c[keep], n[keep] / l2[keep].sqrt()[:, None]], 1).contiguous()


def _dims(case):
    return case["nx"], case["ny"], case["nz"]


def _mesh_input(case, seed):
    v, f = _shape_on_gpu(case["mesh"], case["tris"])
    if case["mode"] == "reference" and case["path"] == "fast":
        # its stratified probes decline some placements: the named one, with vertex noise
        vf, mn, mx = meshgen.fit_to_lattice(_shape(case["mesh"], case["tris"])[0], _dims(case), case["h"])
        return _noisy(torch.from_numpy(vf).to(v.device), 0.02 * case["h"], seed).float(), f, mn, mx
    vf, mn, mx = _place(v, _dims(case), case["h"], seed)
    return vf, f, mn, mx


def _noisy(v, size, seed):
    g = torch.Generator().manual_seed(seed)
    return v + (torch.rand(v.shape, generator=g, dtype=torch.float64) * 2.0 - 1.0).to(v.device) * size


def _noisy_mesh(case, seed):
    """The mesh upright in a lattice whose sides its extent fixes (each extent a whole number
    of voxels, its ends mid-voxel), with vertex noise of up to 0.1 voxel."""
    v, f = _shape_on_gpu(case["mesh"], case["tris"])
    h = case["h"]
    lo, hi = v.min(0).values, v.max(0).values
    s = float(((torch.tensor(_dims(case), device=v.device) - 22) * h / (hi - lo)).min())
    ext = torch.round((hi - lo) * s / h) * h
    v = (v - lo) / (hi - lo) * ext + (torch.round(-ext / (2 * h)) + 0.5) * h
    return _noisy(v, 0.1 * h, seed).float(), f


@functools.lru_cache(maxsize=8)
def _batch_layout(n, layout, t_lo, t_hi, g_lo, g_hi):
    """The uneven meshes of a scene: (kind, triangles, side), fixed by `layout`."""
    r = np.random.RandomState(layout)
    return [(("mug", "vessel", "sphere")[i % 3], int(np.exp(r.uniform(math.log(t_lo), math.log(t_hi)))),
             int(r.randint(g_lo, g_hi + 1))) for i in range(n)]


@functools.lru_cache(maxsize=96)
def _scene_shape(mesh, tris):
    if mesh == "vessel":  # closed tubes, as a scene's clean parts
        levels = int(np.clip(round(math.log2(max(tris, 1) / 3000.0)), 1, 6))
        k = max(1.0, math.sqrt(tris / (2 ** (levels + 1) - 1) / 40.0))
        v, f = meshgen.vessel_tree(seed=tris, levels=levels, around=max(8, round(4 * k)), n_len=max(2, round(3 * k)),
                                   n_cap=max(1, round(k)), defects=False)
    else:
        v, f = _shape(mesh, tris)
    return torch.from_numpy(np.asarray(v, np.float64)).cuda(), torch.from_numpy(np.asarray(f, np.int64)).cuda()


def _field(case, seed):
    """A signed field like an SDF: a thick-walled vessel with a wavy wall and a ring beside it,
    in millimetres, x fastest, each value off by up to 5% (the seed's noise keeps the signs)."""
    ph = (0.3, 1.1, 2.3)
    h = case["h"]
    nx, ny, nz = _dims(case)
    ax = [(torch.arange(n, dtype=torch.float64, device="cuda") - (n - 1) / 2.0 + 0.21) * h for n in (nx, ny, nz)]
    size = min(nx, ny, nz) * h
    out = torch.empty((nz, ny, nx), dtype=torch.float32, device="cuda")
    x, y = ax[0][None, None, :], ax[1][None, :, None]
    for k in range(0, nz, 32):
        z = ax[2][k:k + 32, None, None]
        rad = torch.sqrt(x * x + y * y)
        wave = 0.01 * size * (torch.sin(14.0 * x / size + ph[0]) * torch.sin(11.0 * y / size + ph[1])
                              + torch.sin(17.0 * z / size + ph[2]))
        wall = torch.maximum((rad - 0.3 * size + wave).abs() - 0.03 * size, z.abs() - 0.38 * size)
        ring = torch.sqrt((torch.sqrt((x - 0.33 * size) ** 2 + z * z) - 0.1 * size) ** 2 + y * y) - 0.025 * size
        out[k:k + 32] = torch.minimum(wall, ring).float()
    g = torch.Generator(device="cuda").manual_seed(seed)
    return (out * (0.95 + 0.1 * torch.rand(out.shape, generator=g, device="cuda"))).reshape(-1)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "sdf":
        vf, f, mn, mx = _mesh_input(case, seed)
        tris = _soup(vf, f)
        n = int(np.prod(_dims(case)))
        mem = case["memory"]
        if mem == "device":
            out = torch.zeros(n, dtype=torch.float32, device="cuda")
        else:
            tris = tris.cpu()
            out = torch.zeros(n, dtype=torch.float32, pin_memory=mem == "pinned")
            tris = tris.pin_memory() if mem == "pinned" else tris.numpy()
            out = out if mem == "pinned" else out.numpy()
        kw = {}
        if case["mode"] == "learned":
            kw["mlp_params"] = torch.from_numpy(np.load(learn.MODEL_PATH)["params"]).cuda()
        return dict(kind=kind, tris=tris, h=case["h"], mn=mn, mx=mx, out=out, mode=MODES[case["mode"]],
                    path=PATHS[case["path"]], kw=kw)
    if kind == "build":
        vf, f = _noisy_mesh(case, seed)
        return dict(kind=kind, v=vf.cpu().numpy(), f=f.to(torch.int32).cpu().numpy().astype(np.uint32).ravel(),
                    h=case["h"])
    if kind == "batch":
        meshes, outs = [], []
        layout = _batch_layout(*(case[k] for k in ("n", "layout", "t_lo", "t_hi", "g_lo", "g_hi")))
        for i, (mesh, tris, g) in enumerate(layout):
            v, f = _scene_shape(mesh, tris)
            vf, mn, mx = _place(v, (g, g, g), 1.0, seed * 64 + i, span=0.9)
            meshes.append((_soup(vf, f), 1.0, mn, mx))
            outs.append(torch.zeros(g ** 3, dtype=torch.float32, device="cuda"))
        torch.cuda.synchronize()
        return dict(kind=kind, batch=gbsdf.Batch(meshes, outs=outs, mode=MODES[case["mode"]]), outs=outs)
    if kind == "iso":
        return dict(kind=kind, grid=_field(case, seed), dims=_dims(case), h=case["h"],
                    origin=np.asarray([-n // 2 * case["h"] for n in _dims(case)], np.float32))
    if kind == "file":
        return dict(kind=kind, format=case["format"], data=_file(case, seed))
    X, y, w, p = _rows(case, seed)
    return dict(kind=kind, X=X, y=y, w=w, scale=1.0 / float(w.sum().item()), net=learn.SignRiskMLP(p))


def _file(case, seed):
    v, f = _shape_on_gpu(case["mesh"], case["tris"])
    vf, _, _ = _place(v, (860, 860, 880), 0.1, seed)
    vf, f = vf.cpu().numpy(), f.cpu().numpy()
    if case["format"] == "obj":
        return meshgen.to_obj_text(vf, f, fancy=False)
    return meshgen.to_binary_stl(vf, f) if case["format"] == "stl" else meshgen.to_ascii_stl(vf, f, fancy=False)


def _rows(case, seed):
    """Feature rows in the ranges brick features have, labels and weights as fit() makes
    them, and parameters a few steps from their initial values."""
    n = case["rows"]
    g = torch.Generator().manual_seed(seed)
    X = torch.rand((n, learn.N_FEATURES), generator=g) ** 3 * (torch.rand((n, learn.N_FEATURES), generator=g) < 0.6)
    y = (torch.rand(n, generator=g) < 0.05).float()
    w = torch.where(y > 0.5, 1.0 + torch.randint(1, 60, (n,), generator=g).float(), torch.ones(n))
    p = learn.init_params(seed % 1000) + 0.01 * torch.randn(learn.N_PARAMS, generator=g).numpy()
    return X.cuda(), y.cuda(), w.cuda(), p.astype(np.float32)


# ---- one pass ----------------------------------------------------------------------------
def run(s):
    kind = s["kind"]
    if kind == "sdf":
        out, res = gbsdf.compute_mesh_sdf(s["tris"], s["h"], s["mn"], s["mx"], out=s["out"], mode=s["mode"],
                                          path=s["path"], raise_on_error=False, **s["kw"])
        return {"sdf": out, "status": res.status}
    if kind == "build":
        grid, _ = gbsdf.CudaRasterizer.build_from_mesh(s["v"], s["f"], s["h"])
        return {"sdf": grid.data, "min": grid.min_coord, "dims": grid.dims}
    if kind == "batch":
        statuses, _ = s["batch"].run()
        return {"sdf": list(s["outs"]), "status": list(statuses)}
    if kind == "iso":
        v, i = gbsdf.extract_iso_surface(s["grid"], s["dims"], s["h"], s["origin"], 0.0, outputs_on_device=True)
        return {"vertices": v, "indices": i}
    if kind == "file":
        if s["format"] == "obj":
            v, i = gbsdf.parse_obj(s["data"])
            i, orientable, _, _, _ = gbsdf.orient_mesh(v, i)
        else:
            v, i, orientable = gbsdf.parse_stl(s["data"])
        return {"vertices": v, "indices": i, "orientable": orientable}
    g, loss = s["net"].grad(s["X"], s["y"], s["w"])
    s["net"].adam(g, lr=2e-3, scale=s["scale"])
    return {"grad": g, "loss": loss, "params": s["net"].P, "logits": s["net"].logits(s["X"])}


# ---- what a pass cannot do without -------------------------------------------------------
def work(case):
    kind = case["kind"]
    if kind == "sdf":
        return _build_work(np.prod(_dims(case)), case["tris"], case["path"] == "fast" or np.prod(_dims(case)) >= 1 << 25)
    if kind == "build":
        return _build_work(np.prod(_dims(case)), case["tris"], False)
    if kind == "batch":
        layout = _batch_layout(*(case[k] for k in ("n", "layout", "t_lo", "t_hi", "g_lo", "g_hi")))
        each = [_build_work(g ** 3, t, True) for _, t, g in layout]
        return {k: sum(w[k] for w in each) for k in ("bytes", "flops")}
    if kind == "iso":
        cells = float(min(_dims(case))) ** 2  # crossed cells, about: 3.5 areas of the smallest side
        return {"bytes": 4.0 * np.prod(_dims(case)) + 3.5 * cells * (12 + 24), "flops": 3.5 * cells * 20}
    if kind == "file":
        per = {"stl": 50, "ascii_stl": 222, "obj": 36}[case["format"]]
        return {"bytes": case["tris"] * (per + 12.0 + 6.0), "flops": 0.0}
    return {"bytes": case["rows"] * (4.0 * learn.N_FEATURES + 12) + 16.0 * learn.N_PARAMS,
            "flops": case["rows"] * 4.0 * 2 * (32 * 64 + 64 * 64 + 64)}


def _build_work(n, tris, fast):
    """Triangles in, grid out; on the fast path the 48 sweeps' updates (about 25 operations a
    voxel and sweep), else one exact distance (60 operations) and one sign a voxel."""
    return {"bytes": 4.0 * n + 48.0 * tris, "flops": (48 * 25.0 if fast else 60.0) * n}


# ---- the same in 64 bits -----------------------------------------------------------------
EXACT_VOXELS = 4_500_000


def exact(case, seed):
    kind = case["kind"]
    if kind in ("sdf", "build"):
        n = int(np.prod(_dims(case)))
        closed = case["mesh"] in ("mug", "sphere")
        fast = kind == "sdf" and case["path"] == "fast"
        if fast and case["mode"] == "reference":
            return None  # the probes' patches are part of its result
        if not closed or n > EXACT_VOXELS or (not fast and n * case["tris"] > 4e8):
            return None
        if kind == "build":
            return None  # its lattice is the library's own
        vf, f, mn, _ = _mesh_input(case, seed)
        tris = _soup(vf, f).double()
        d = _distance(tris, case["h"], mn, _dims(case), 8 if fast else None)
        if fast:
            d = _converged(d, case["h"]) if case["mode"] == "exact" else _swept(d, case["h"])
        d = torch.where(_inside(tris, case["h"], mn, _dims(case)), -d, d).reshape(-1)
        return {"sdf": d if case["memory"] == "device" else d.cpu(), "status": 0}
    if kind == "iso":
        g = _field(case, seed).double()
        return {"vertices": _crossings(g, _dims(case), case["h"], [-n // 2 * case["h"] for n in _dims(case)]),
                "indices": None}
    if kind == "file" and case["format"] == "stl":
        return {"vertices": _welded(_file(case, seed)), "indices": None, "orientable": None}
    if kind == "train":
        return _step(case, seed)
    return None


def _h32(h):
    return float(np.float32(h))


def _distance(tris, h, mn, dims, band):
    """Distance of each voxel to the nearest triangle; with `band`, only within that many
    voxels (infinite elsewhere). Sub-array [z, y, x]."""
    h = _h32(h)
    nx, ny, nz = dims
    best = torch.full((nz * ny * nx,), math.inf, dtype=torch.float64, device=tris.device)
    v = tris[:, :9].reshape(-1, 3, 3)
    dim = torch.tensor([nx, ny, nz], device=tris.device)
    low = torch.tensor(mn.astype(np.int64), device=tris.device)
    if band is None:
        b0 = torch.zeros((len(v), 3), dtype=torch.int64, device=tris.device)
        b1 = (dim - 1).expand(len(v), 3)
    else:
        b0 = torch.maximum(torch.floor(v.amin(1) / h - band).long() - low, torch.zeros_like(dim))
        b1 = torch.minimum(torch.ceil(v.amax(1) / h + band).long() - low, dim - 1)
    size = (b1 - b0 + 1).clamp(min=0)
    count = size.prod(1)
    ends = count.cumsum(0)
    at = 0
    while at < len(v):
        stop = int(torch.searchsorted(ends, (ends[at - 1] if at else 0) + 6_000_000, right=True))
        stop = min(max(stop, at + 1), len(v))
        c = count[at:stop]
        t = torch.repeat_interleave(torch.arange(at, stop, device=v.device), c)
        k = torch.arange(len(t), device=v.device) - torch.repeat_interleave(c.cumsum(0) - c, c)
        sx, sy = size[t, 0], size[t, 1]
        x, y, z = b0[t, 0] + k % sx, b0[t, 1] + k // sx % sy, b0[t, 2] + k // (sx * sy)
        p = torch.stack([x + low[0], y + low[1], z + low[2]], 1).double() * h
        d = _point_triangle(p, v[t, 0], v[t, 1], v[t, 2])
        best.scatter_reduce_(0, (z * ny + y) * nx + x, d, "amin")
        at = stop
    if band is not None:
        best = torch.where(best <= band * h, best, math.inf)
    return best.reshape(nz, ny, nx)


def _point_triangle(p, a, b, c):
    """Distance of points to triangles: to the plane where the foot is inside, else to the
    nearest of the three edges."""
    n = torch.linalg.cross(b - a, c - a)
    nn = (n * n).sum(1)
    inside = nn > 0
    edge = torch.full_like(nn, math.inf)
    for u, w in ((a, b), (b, c), (c, a)):
        e, q = w - u, p - u
        s = ((q * e).sum(1) / (e * e).sum(1).clamp(min=1e-300)).clamp(0.0, 1.0)
        edge = torch.minimum(edge, ((q - s[:, None] * e) ** 2).sum(1))
        inside = inside & ((torch.linalg.cross(e, q) * n).sum(1) >= 0)
    plane = ((p - a) * n).sum(1) ** 2 / nn.clamp(min=1e-300)
    return torch.where(inside, torch.minimum(plane, edge), edge).sqrt()


def _inside(tris, h, mn, dims):
    """Inside by signed crossings of the upward ray through each column (closed meshes)."""
    h = _h32(h)
    nx, ny, nz = dims
    v = tris[:, :9].reshape(-1, 3, 3)
    low = torch.tensor(mn.astype(np.int64), device=v.device)
    dim = torch.tensor(dims, device=v.device)
    b0 = torch.maximum(torch.ceil(v.amin(1) / h).long() - low, torch.zeros_like(dim))[:, :2]
    b1 = torch.minimum(torch.floor(v.amax(1) / h).long() - low, dim - 1)[:, :2]
    size = (b1 - b0 + 1).clamp(min=0)
    c = size.prod(1)
    t = torch.repeat_interleave(torch.arange(len(v), device=v.device), c)
    k = torch.arange(len(t), device=v.device) - torch.repeat_interleave(c.cumsum(0) - c, c)
    x, y = b0[t, 0] + k % size[t, 0], b0[t, 1] + k // size[t, 0]
    px, py = (x + low[0]).double() * h + 1e-9 * h, (y + low[1]).double() * h + 1.7e-9 * h
    A, B, C = v[t, 0], v[t, 1], v[t, 2]

    def side(p, q):
        return (q[:, 0] - p[:, 0]) * (py - p[:, 1]) - (q[:, 1] - p[:, 1]) * (px - p[:, 0])

    wa, wb, wc = side(B, C), side(C, A), side(A, B)
    up, down = (wa > 0) & (wb > 0) & (wc > 0), (wa < 0) & (wb < 0) & (wc < 0)
    hit = up | down
    z = (wa * A[:, 2] + wb * B[:, 2] + wc * C[:, 2]) / (wa + wb + wc)
    below = torch.ceil(z / h).long() - low[2]  # voxels under the crossing: z index < below
    hit = hit & (below > 0)
    turn = torch.zeros((nz + 1) * ny * nx, dtype=torch.int32, device=v.device)
    turn.index_add_(0, ((below.clamp(max=nz) * ny + y) * nx + x)[hit],
                    torch.where(up, 1, -1).to(torch.int32)[hit])
    w = turn.reshape(nz + 1, ny, nx).flip(0).cumsum(0).flip(0)[1:]
    return w != 0


def _sweeps(u, update):
    """One round: six sweeps, each line by line with its neighbour lines as they were when
    the sweep began."""
    far = 1e30
    for axis in (2, 1, 0):
        others = [a for a in (0, 1, 2) if a != axis]
        for step in (1, -1):
            old = u
            u = u.clone()
            n = u.shape[axis]
            side = []
            for a in others:
                pad = torch.full_like(old.narrow(a, 0, 1), far)
                side.append(torch.minimum(torch.cat([pad, old.narrow(a, 0, old.shape[a] - 1)], a),
                                          torch.cat([old.narrow(a, 1, old.shape[a] - 1), pad], a)))
            prev = None
            for i in range(n) if step > 0 else range(n - 1, -1, -1):
                o = old.select(axis, i)
                nxt = old.select(axis, i + step) if 0 <= i + step < n else torch.full_like(o, far)
                along = nxt if prev is None else torch.minimum(prev, nxt)
                prev = torch.minimum(o, update(along, side[0].select(axis, i), side[1].select(axis, i)))
                u.select(axis, i).copy_(prev)
    return u


def _sorted3(a, b, c):
    s0, s2 = torch.minimum(a, torch.minimum(b, c)), torch.maximum(a, torch.maximum(b, c))
    return s0, torch.maximum(torch.minimum(a, b), torch.minimum(torch.maximum(a, b), c)), s2


def _swept(u, h):
    """Eight rounds of the update with the halved 3D pairwise sum."""
    h = _h32(h)
    u = u.clamp(max=1e30)

    def update(a, b, c):
        s0, s1, s2 = _sorted3(a, b, c)
        d2 = 2 * h * h - (s1 - s0) ** 2
        d3 = 3 * h * h - 0.5 * ((s1 - s0) ** 2 + (s2 - s1) ** 2 + (s2 - s0) ** 2)
        u1 = s0 + h
        u2 = (s0 + s1 + d2.clamp(min=0).sqrt()) / 2
        u3 = (s0 + s1 + s2 + d3.clamp(min=0).sqrt()) / 3
        two = (u1 > s1) & (d2 >= 0)
        return torch.where(two & (u2 > s2) & (d3 >= 0), u3, torch.where(two, u2, u1))

    for _ in range(8):
        u = _sweeps(u, update)
    return u


def _converged(u, h):
    """The corrected update to its fixed point."""
    h = _h32(h)
    u = u.clamp(max=1e30)

    def update(a, b, c):
        s0, s1, s2 = _sorted3(a, b, c)
        p, q = s1 - s0, s2 - s0
        u1 = torch.full_like(s0, h)
        u2 = (p + (2 * h * h - p * p).clamp(min=0).sqrt()) / 2
        u3 = (p + q + (3 * h * h - p * p - q * q - (q - p) ** 2).clamp(min=0).sqrt()) / 3
        return s0 + torch.where(u1 <= p, u1, torch.where(u2 <= q, u2, u3))

    for _ in range(48):
        new = _sweeps(u, update)
        done = bool(((u - new).abs() <= 1e-9 * h).all())
        u = new
        if done:
            break
    return u


def _crossings(g, dims, h, origin):
    """One vertex on each crossed grid edge, in voxel order (x, y, z edges of a voxel in
    turn); voxels of the grid's border are outside by at least one voxel size."""
    h = _h32(h)
    nx, ny, nz = dims
    g = g.reshape(nz, ny, nx).clone()
    for a in range(3):
        for i in (0, g.shape[a] - 1):
            g.select(a, i).clamp_(min=h)
    found = []
    for k in range(3):  # k = 0, 1, 2: edges along x, y, z, i.e. axes 2, 1, 0
        a = 2 - k
        u, w = g.narrow(a, 0, g.shape[a] - 1), g.narrow(a, 1, g.shape[a] - 1)
        z, y, x = torch.nonzero((u <= 0) != (w <= 0), as_tuple=True)
        p, q = u[z, y, x], w[z, y, x]
        at = torch.stack([x, y, z], 1).double()
        at[:, k] += p / (p - q)
        found.append((((z * ny + y) * nx + x) * 3 + k, at))
    key, at = (torch.cat([f[j] for f in found]) for j in (0, 1))
    start = torch.tensor([float(np.float32(o)) for o in origin], dtype=torch.float64, device=g.device)
    return start + at[key.argsort()] * h


def _welded(data):
    """The distinct corners of a binary STL (by coordinates rounded to 1e-4), first seen first."""
    n = int(np.frombuffer(data[80:84], np.uint32)[0])
    rec = np.frombuffer(data[84:84 + 50 * n], np.dtype([("n", "<f4", 3), ("v", "<f4", (3, 3)), ("a", "<u2")]))
    c = rec["v"].reshape(-1, 3)
    key = np.rint(c * np.float32(10000.0)).astype(np.int64)
    _, first = np.unique(key, axis=0, return_index=True)
    return c[np.sort(first)].astype(np.float64)


def _step(case, seed):
    """Weighted cross-entropy gradient summed over the rows, one Adam step, the new scores."""
    X, y, w, p = (t.double() if isinstance(t, torch.Tensor) else torch.from_numpy(t).double().cuda()
                  for t in _rows(case, seed))
    scale = 1.0 / float(w.float().sum().item())

    def scores(q):
        w1, b1, w2, b2, w3, b3 = torch.split(q, [64 * 32, 64, 64 * 64, 64, 64, 1])
        a = torch.relu(X @ w1.reshape(64, 32).T + b1)
        return torch.relu(a @ w2.reshape(64, 64).T + b2) @ w3 + b3

    p = p.clone().requires_grad_(True)
    loss = (w * torch.nn.functional.binary_cross_entropy_with_logits(scores(p), y, reduction="none")).sum()
    g, = torch.autograd.grad(loss, p)
    with torch.no_grad():
        s = g * scale
        m, v = 0.1 * s, 0.001 * s * s
        new = p - 2e-3 * (m / 0.1) / ((v / 0.001).sqrt() + 1e-8)
        return {"grad": g, "loss": float(loss), "params": new, "logits": scores(new)}
