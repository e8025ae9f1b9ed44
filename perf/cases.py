"""Measured cases of the distance-field library, through its public entry points.

A case is a dict of plain values; ``kind`` says which entry point it goes through, ``mesh`` and
``detail`` the surface (``workloads``' generators at a size), the rest the query:

* ``grid``        signed / unsigned node grid on a resident mesh (``DeviceMesh.query_grid``)
* ``points``      point list on a resident mesh (``DeviceMesh.query_points``)
* ``batch``       uneven meshes, each with a grid or a point list, in one launch (``Batch``)
* ``moving``      a surface that moves: mesh built from device arrays, queried once, dropped
* ``call_grid``   blocking drop-in call from host arrays (``sample_sdf_bvh``)
* ``call_points`` blocking drop-in call from host arrays (``edf_select``, ``closest_point_bvh``)
* ``radius``      closest triangle or quad within a radius, host arrays (``closest_within_radius``)
* ``pairs``       candidate contact pairs, host arrays (``potential_contact``)
* ``round``       a field rounded by a radius, host arrays (``round_sdf``)
* ``dense``       the plain methods on device arrays (``edf_device``: brute force, cell list)

``precision`` is the query arithmetic: ``fixup`` (float traversal, double result), ``f64``, ``f32``.
"""

import math

import numpy as np
import torch

import ssdf_b200 as S
from ssdf_b200 import workloads as W

PRECISION = {"fixup": 2, "f64": 1, "f32": 0}  # SSDF_PREC_*
OUTPUT = {"edf": 0, "sqedf": 1, "sdf": 2, "closest": 3}  # SSDF_OUT_*

# Point-triangle pairs up to which the 64-bit answer is computed pair by pair.
EXACT_PAIRS = 8_000_000_000


def listed():
    return [
        # a control loop's probes or a contact search's few nodes against a small resident surface
        dict(name="points_few", kind="points", mesh="icosphere", detail=3, n=1000, where="box", precision="fixup",
             output="sdf"),
        # the benchmark's small grid: signed distances and closest triangles of a 64^3 cell-centred grid
        dict(name="grid_icosphere_64", kind="grid", mesh="icosphere", detail=4, nx=64, ny=64, nz=64, pad=0.2,
             precision="fixup", output="sdf"),
        # the benchmark's default grid: 256^3 signed nodes around a 131,072-triangle closed surface
        dict(name="grid_knot_256", kind="grid", mesh="knot", detail=1024, nx=256, ny=256, nz=256, pad=0.25,
             precision="fixup", output="sdf"),
        # a ragged grid in plain double arithmetic
        dict(name="grid_torus_f64", kind="grid", mesh="torus", detail=203, nx=131, ny=97, nz=61, pad=0.3,
             precision="f64", output="edf"),
        # the benchmark's float point cloud around an open, overlapping lattice of thin beams
        dict(name="points_beams_f32", kind="points", mesh="beams", detail=20000, n=4_000_000, where="box",
             precision="f32", output="edf"),
        # particles near a surface: a simulation's scattered points, signed
        dict(name="points_near_knot", kind="points", mesh="knot", detail=1024, n=500_003, where="near",
             precision="fixup", output="sdf"),
        # many parts at once: uneven meshes with grids and point lists, one launch
        dict(name="batch_parts", kind="batch", meshes=12, layout=7, tri_lo=1000, tri_hi=60000, side_lo=24, side_hi=80),
        # a fluid-structure step: the surface has moved, build it from device arrays and query it once
        dict(name="moving_torus", kind="moving", mesh="torus", detail=256, n=100_000, where="near",
             precision="fixup", output="sdf"),
        # the drop-in call of a program that keeps its arrays on the host
        dict(name="call_grid_96", kind="call_grid", mesh="icosphere", detail=5, nx=96, ny=96, nz=96, pad=0.2),
        # the closest triangle within a search radius, for contact detection
        dict(name="radius_knot", kind="radius", mesh="knot", detail=512, n=200_000, reach=0.05, quads=False),
        # a level set's corners rounded, from a sampled field
        dict(name="round_box_72", kind="round", n=72, radius=0.1),
        # the plain cell-list method a program selects explicitly
        dict(name="dense_celllist", kind="dense", mesh="icosphere", detail=4, n=150_001, where="box", method=1,
             precision="f64"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_mesh(rng, most):
    mesh = rng.choice(["icosphere", "torus", "knot", "beams"])
    if mesh == "icosphere":
        return dict(mesh=mesh, detail=rng.randint(2, 5 if most < 60000 else 6))
    if mesh == "beams":
        return dict(mesh=mesh, detail=_log_int(rng, 80, most // 12))
    return dict(mesh=mesh, detail=_log_int(rng, 24, int(math.sqrt(most / 2 * (2 if mesh == "torus" else 16)))))


def draw(rng):
    kind = rng.choice(["grid", "grid", "points", "points", "batch", "moving", "call_grid", "call_points", "radius",
                       "pairs", "round", "dense"])
    if kind == "grid":
        c = dict(kind=kind, **_draw_mesh(rng, 131072))
        side = math.exp(rng.uniform(math.log(20), math.log(170)))
        for k in ("nx", "ny", "nz"):
            c[k] = max(2, int(side * rng.uniform(0.6, 1.5)))
        c.update(pad=rng.uniform(0.05, 0.4), precision=rng.choice(["fixup", "fixup", "f64"]),
                 output=rng.choice(["sdf", "sdf", "edf"]))
        return c
    if kind == "points":
        c = dict(kind=kind, **_draw_mesh(rng, 131072), n=_log_int(rng, 100, 2_000_000))
        c.update(where=rng.choice(["box", "near"]), precision=rng.choice(["fixup", "fixup", "f64", "f32"]))
        c["output"] = "edf" if c["precision"] == "f32" else rng.choice(["sdf", "edf"])
        return c
    if kind == "batch":
        return dict(kind=kind, meshes=rng.randint(3, 12), layout=rng.randrange(1 << 20), tri_lo=rng.randint(300, 2000), tri_hi=_log_int(rng, 4000, 60000),
                    side_lo=rng.randint(12, 32), side_hi=rng.randint(33, 80))
    if kind == "moving":
        return dict(kind=kind, **_draw_mesh(rng, 131072), n=_log_int(rng, 1000, 500_000), where="near",
                    precision="fixup", output="sdf")
    if kind == "call_grid":
        c = dict(kind=kind, **_draw_mesh(rng, 60000))
        side = math.exp(rng.uniform(math.log(16), math.log(110)))
        for k in ("nx", "ny", "nz"):
            c[k] = max(2, int(side * rng.uniform(0.7, 1.4)))
        c["pad"] = rng.uniform(0.05, 0.4)
        return c
    if kind == "call_points":
        return dict(kind=kind, **_draw_mesh(rng, 131072), n=_log_int(rng, 200, 1_000_000),
                    where=rng.choice(["box", "near"]), precision=rng.choice(["f64", "f32"]),
                    output=rng.choice(["edf", "closest"]))
    if kind == "radius":
        quads = rng.random() < 0.4
        c = dict(kind=kind, n=_log_int(rng, 500, 500_000), reach=rng.uniform(0.005, 0.2), quads=quads)
        c.update(dict(mesh="torus", detail=_log_int(rng, 24, 256)) if quads else _draw_mesh(rng, 100000))
        return c
    if kind == "pairs":
        return dict(kind=kind, mesh=rng.choice(["torus", "knot"]), detail=_log_int(rng, 40, 512),
                    reach=rng.uniform(0.002, 0.03))
    if kind == "round":
        return dict(kind=kind, n=rng.randint(20, 72), radius=rng.uniform(0.04, 0.12))
    method = rng.randint(0, 1)
    c = dict(kind="dense", **_draw_mesh(rng, 20000), n=_log_int(rng, 500, 150_000), where=rng.choice(["box", "near"]),
             method=method, precision=rng.choice(["f64", "f32"]))
    if method == 0:  # every pair is tested: keep the pairs below 2^31
        c["n"] = min(c["n"], max(500, (1 << 31) // max(1, _triangles(c))))
    return c


# ---- inputs -----------------------------------------------------------------------------------------

def _mesh(case, seed):
    """The surface of a case. The seed moves its vertices (or beams); the size is the case's."""
    d = int(case["detail"])
    if case["mesh"] == "icosphere":
        return W.icosphere(d, seed=seed)
    if case["mesh"] == "torus":
        return W.torus(nu=d, nv=max(3, d // 2), jitter=0.01, seed=seed)
    if case["mesh"] == "knot":
        return W.torus_knot_tube(nu=d, nv=max(3, d // 16), seed=seed)
    return W.beam_lattice(d, seed=seed)


def _triangles(case):
    d = int(case["detail"])
    if case["mesh"] == "icosphere":
        return 20 * 4 ** d
    if case["mesh"] == "torus":
        return 2 * d * max(3, d // 2)
    if case["mesh"] == "knot":
        return 2 * d * max(3, d // 16)
    return 12 * d


def _vertices(case):
    return _triangles(case) // 2 if case["mesh"] != "beams" else 8 * int(case["detail"])


def _points(case, mesh, seed):
    """(3, n) float64 on the GPU: uniform in the padded box, or scattered around the surface."""
    g = torch.Generator(device="cuda").manual_seed(int(seed) % (1 << 31) + 17)
    n = int(case["n"])
    lo, hi = (torch.tensor(v, device="cuda") for v in mesh.bbox())
    if case.get("where") == "near":
        v = torch.from_numpy(mesh.vertices).cuda()
        t = torch.from_numpy(mesh.triangles).cuda().long()
        pick = t[torch.randint(0, mesh.nt, (n,), generator=g, device="cuda")]
        w = torch.rand((n, 2), generator=g, device="cuda", dtype=torch.float64)
        w = torch.where(w.sum(1, keepdim=True) > 1, 1 - w, w)
        a, b, c = v[pick[:, 0]], v[pick[:, 1]], v[pick[:, 2]]
        p = a + w[:, :1] * (b - a) + w[:, 1:] * (c - a)
        p = p + 0.02 * torch.randn((n, 3), generator=g, device="cuda", dtype=torch.float64)
    else:
        pad = 0.1 * (hi - lo)
        p = (lo - pad) + (hi - lo + 2 * pad) * torch.rand((n, 3), generator=g, device="cuda", dtype=torch.float64)
    return p.t().contiguous()


def _grid(case, mesh):
    lo, hi = mesh.bbox()
    pad = float(case["pad"])
    return W.Grid((int(case["nx"]), int(case["ny"]), int(case["nz"])), tuple(float(v) for v in lo - pad),
                  tuple(float(v) for v in hi + pad))


def _dtype(case):
    return torch.float32 if case.get("precision") == "f32" else torch.float64


def _parts(case, seed):
    """The batch's meshes and grids: shapes and sizes by the case's layout, scaled, moved and jittered by
    the seed."""
    r = np.random.default_rng(seed)
    parts = []
    for mesh, grid in W.multi_mesh_set(int(case["meshes"]), float(case["tri_lo"]), float(case["tri_hi"]),
                                       float(case["side_lo"]), float(case["side_hi"]), seed=int(case["layout"])):
        v = mesh.vertices * r.uniform(0.8, 1.25) + r.uniform(-0.5, 0.5, size=3)
        m = W.Mesh(v + 1e-4 * mesh.diagonal() * r.uniform(-1.0, 1.0, size=v.shape), mesh.triangles)
        parts.append((m, W.Grid.padded_nodes(m, int(grid.n[0]), 0.1 * m.diagonal())))
    return parts


def _field(case, seed):
    """A box with randomly placed faces sampled on a uniform grid, positive inside."""
    r = np.random.default_rng(seed)
    n = int(case["n"])
    half = 0.45 + 0.1 * r.random(3)
    centre = 0.04 * (r.random(3) - 0.5)
    h = 2.0 / (n - 1)
    x = -1.0 + h * np.arange(n)
    q = [np.abs(x - centre[d]) - half[d] for d in range(3)]
    qx, qy, qz = q[0][None, None, :], q[1][None, :, None], q[2][:, None, None]
    outside = np.sqrt(np.maximum(qx, 0) ** 2 + np.maximum(qy, 0) ** 2 + np.maximum(qz, 0) ** 2)
    inside = np.minimum(np.maximum(np.maximum(qx, qy), qz), 0.0)
    return S.GridGeometry((n, n, n), (-1.0, -1.0, -1.0), (h, h, h)), -(outside + inside).ravel()


def _quads(mesh):
    """The torus' quads from its triangle pairs: (a, b, d) and (a, d, c) of one cell, either winding."""
    half = mesh.nt // 2
    t0, t1 = mesh.triangles[:half], mesh.triangles[half:]
    if np.array_equal(t0[:, 2], t1[:, 1]):  # (a, b, d), (a, d, c)
        cols = [t0[:, 0], t0[:, 1], t0[:, 2], t1[:, 2]]
    else:  # wound the other way: (a, d, b), (a, c, d)
        cols = [t0[:, 0], t1[:, 1], t1[:, 2], t0[:, 2]]
    return [np.ascontiguousarray(c, dtype=np.int32) for c in cols]


def prepare(case, seed):
    kind = case["kind"]
    st = {"case": case}
    if kind == "batch":
        parts = _parts(case, seed)
        batch = S.Batch(len(parts))
        batch.reserve(sum(g.size for _, g in parts))
        st.update(batch=batch, outs=[], keep=[])
        for k, (mesh, grid) in enumerate(parts):  # every third one at points scattered around its surface
            dm = S.DeviceMesh(mesh)
            n = grid.size
            out = torch.empty(n, device="cuda", dtype=torch.float64)
            tri = torch.empty(n, device="cuda", dtype=torch.int32)
            if k % 3 == 2:
                p = _points(dict(n=n, where="near"), mesh, seed + k)
                batch.add_points(dm, p[0], p[1], p[2], out, tri)
                st["keep"].append((dm, p))
            else:
                batch.add_grid(dm, grid, out, tri)
                st["keep"].append(dm)
            st["outs"] += [out, tri]
        return st
    if kind == "round":
        st["grid"], st["f"] = _field(case, seed)
        return st
    mesh = _mesh(case, 1 if kind == "pairs" else seed)
    if kind == "grid":
        grid = _grid(case, mesh)
        st.update(mesh=S.DeviceMesh(mesh, normals=case["output"] == "sdf"), grid=grid,
                  out=torch.empty(grid.size, device="cuda", dtype=torch.float64),
                  tri=torch.empty(grid.size, device="cuda", dtype=torch.int32))
    elif kind in ("points", "moving", "dense"):
        dt = _dtype(case)
        p = _points(case, mesh, seed).to(dt)
        n = p.shape[1]
        st.update(p=p, out=torch.empty(n, device="cuda", dtype=dt), tri=torch.empty(n, device="cuda", dtype=torch.int32))
        if kind == "points":
            st["mesh"] = S.DeviceMesh(mesh, np.float32 if case["precision"] == "f32" else np.float64,
                                      keep_fp64=case["precision"] != "f32", normals=case["output"] == "sdf")
        else:
            st["idx"] = [torch.from_numpy(a).cuda() for a in mesh.indices()]
            st["xyz"] = [torch.from_numpy(a).cuda().to(dt) for a in mesh.coords()]
    elif kind == "call_grid":
        st.update(mesh=mesh, grid=_grid(case, mesh))
    elif kind == "call_points":
        st.update(mesh=mesh, p=_points(case, mesh, seed).to(_dtype(case)).cpu().numpy())
    elif kind == "radius":
        st.update(p=_points(dict(n=case["n"], where="near"), mesh, seed).cpu().numpy(), vertices=mesh.coords(),
                  elements=_quads(mesh) if case["quads"] else mesh.indices(),
                  r2=np.array([float(case["reach"]) ** 2]))
    elif kind == "pairs":  # one surface, its elements in an order of the seed's (so the pairs' number is the case's)
        order = np.random.default_rng(seed).permutation(mesh.nt)
        st.update(vertices=mesh.coords(), elements=[np.ascontiguousarray(a[order]) for a in mesh.indices()])
    return st


# ---- one pass ---------------------------------------------------------------------------------------

def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "batch":
        st["batch"].run()
        return st["outs"]
    if kind == "round":
        r = float(case["radius"])
        return S.round_sdf(st["grid"], st["f"], r, 4.0 * r)
    if kind == "call_grid":
        return S.sample_sdf_bvh(st["mesh"], st["grid"])
    if kind == "call_points":
        dt = np.float32 if case["precision"] == "f32" else np.float64
        if case["output"] == "closest":
            return S.closest_point_bvh(st["p"], st["mesh"], dtype=dt)
        return S.edf_select(st["p"], st["mesh"], dtype=dt)
    if kind == "radius":
        return S.closest_within_radius(st["p"], st["elements"], st["vertices"], st["r2"], stride=0)
    if kind == "pairs":
        return S.potential_contact(st["elements"], st["vertices"], float(case["reach"]))
    out, tri = st["out"], st["tri"]
    prec = PRECISION[case["precision"]]
    code = S.F32 if case["precision"] == "f32" else S.F64
    unsigned = kind == "dense" or case["output"] == "edf"
    if unsigned:  # in/out: the caller's bound, here none
        out.fill_(torch.finfo(out.dtype).max)
    if kind == "grid":
        st["mesh"].query_grid(st["grid"], out, tri, precision=prec, output=OUTPUT[case["output"]])
    elif kind == "points":
        st["mesh"].query_points(*st["p"], out, tri, precision=prec, output=OUTPUT[case["output"]], coord_type=code,
                                out_type=code)
    elif kind == "moving":
        mesh = S.DeviceMesh.from_device(*st["idx"], *st["xyz"], normals=True)
        mesh.query_points(*st["p"], out, tri, precision=prec, output=OUTPUT[case["output"]], coord_type=code,
                          out_type=code)
        mesh.close()
    else:
        S.edf_device(int(case["method"]), *st["p"], *st["idx"], *st["xyz"], out, tri)
    return out, tri


# ---- what a pass cannot do without ------------------------------------------------------------------

def work(case):
    """Bytes: every input read and every output written once (resident meshes' vertices and indices
    included). Operations: one point-triangle distance (79) per query, the least that gives an answer, or
    one box test (6) per element where the answer is a set of pairs."""
    kind = case["kind"]
    if kind == "batch":
        parts = int(case["meshes"])
        tri = math.sqrt(float(case["tri_lo"]) * float(case["tri_hi"])) * parts
        # sides are log-uniform: the mean of side^3
        a, b = float(case["side_lo"]), float(case["side_hi"])
        n = parts * (b ** 3 - a ** 3) / (3 * math.log(b / a))
        return {"bytes": n * 12 + tri * 24, "flops": 79.0 * n}
    if kind == "round":
        n = float(case["n"]) ** 3
        return {"bytes": 16 * n, "flops": 79.0 * 3 * n}
    w = 4 if case.get("precision") == "f32" else 8
    nt, nv = _triangles(case), _vertices(case)
    surface = 12 * nt + 3 * w * nv
    if kind == "pairs":
        return {"bytes": surface + 8 * nt, "flops": 6.0 * nt}
    if kind in ("grid", "call_grid"):
        n = int(case["nx"]) * int(case["ny"]) * int(case["nz"])
        per = 8 + (4 if kind == "grid" else 0)
    else:
        n = int(case["n"])
        per = 3 * w + {"radius": 4 * w + 4, "call_points": 4 * w + 4 if case.get("output") == "closest" else w}.get(
            kind, w + 4)
    return {"bytes": surface + per * n, "flops": 79.0 * n}


# ---- the same in 64 bits ------------------------------------------------------------------------------

def _closest(p, a, b, c):
    """Closest points (rows x columns) of points p to triangles abc and their squared distances: the
    nearest of the three edges' closest points, or the foot on the plane where it lies inside."""
    def dot(u, v):
        return (u * v).sum(-1)

    p = p[:, None, :]
    a, b, c = a[None], b[None], c[None]
    n = torch.linalg.cross(b - a, c - a)
    nn = dot(n, n)
    foot = p - n * (dot(p - a, n) / nn)[..., None]
    inside = nn > 0
    best, at = None, None
    for u, v in ((a, b), (b, c), (c, a)):
        e = v - u
        inside = inside & (dot(torch.linalg.cross(e.expand_as(foot), foot - u), n.expand_as(foot)) >= 0)
        t = (dot(p - u, e) / dot(e, e).clamp_min(1e-300)).clamp(0, 1)
        q = u + t[..., None] * e
        d = dot(p - q, p - q)
        best, at = (d, q) if best is None else (torch.minimum(best, d), torch.where((d < best)[..., None], q, at))
    d = dot(p - foot, p - foot)
    return torch.where(inside, d, best), torch.where(inside[..., None], foot, at)


def _solid_angles(p, a, b, c):
    u, v, w = a[None] - p[:, None], b[None] - p[:, None], c[None] - p[:, None]
    lu, lv, lw = u.norm(dim=-1), v.norm(dim=-1), w.norm(dim=-1)
    num = (u * torch.linalg.cross(v, w)).sum(-1)
    den = lu * lv * lw + (u * v).sum(-1) * lw + (v * w).sum(-1) * lu + (w * u).sum(-1) * lv
    return 2 * torch.atan2(num, den)


def _exact_distances(p, mesh, dtype, signed):
    """Distances (negative inside where signed) and closest points of the (3, n) points p, pair by pair.
    Vertices are rounded to dtype, as the query reads them."""
    v = torch.from_numpy(mesh.vertices).cuda().to(dtype).double()
    t = torch.from_numpy(mesh.triangles).cuda().long()
    a, b, c = v[t[:, 0]], v[t[:, 1]], v[t[:, 2]]
    p = p.double().t()
    rows = max(1, (1 << 23) // max(1, min(mesh.nt, 1 << 13)))
    dist, at = [], []
    for r in range(0, p.shape[0], rows):
        q = p[r:r + rows]
        best = torch.full((q.shape[0],), math.inf, device="cuda", dtype=torch.float64)
        foot, wind = torch.zeros_like(q), torch.zeros_like(best)
        for s in range(0, mesh.nt, 1 << 13):
            tri = [x[s:s + (1 << 13)] for x in (a, b, c)]
            d, f = _closest(q, *tri)
            m, k = d.min(1)
            foot = torch.where((m < best)[:, None], f[torch.arange(len(q), device="cuda"), k], foot)
            best = torch.minimum(best, m)
            if signed:
                wind += _solid_angles(q, *tri).sum(1)
        d = best.sqrt()
        dist.append(torch.where(wind > 2 * math.pi, -d, d) if signed else d)
        at.append(foot)
    return torch.cat(dist), torch.cat(at)


def exact(case, seed):
    kind = case["kind"]
    if kind in ("batch", "round", "pairs") or case.get("quads"):
        return None
    n = int(case["nx"]) * int(case["ny"]) * int(case["nz"]) if "nx" in case else int(case["n"])
    if n * _triangles(case) > EXACT_PAIRS:
        return None
    signed = kind == "call_grid" or case.get("output") == "sdf"
    if signed and case["mesh"] == "beams":
        return None  # overlapping beams: the winding number counts them, the nearest face decides the sign
    mesh = _mesh(case, seed)
    dt = _dtype(case)
    if "nx" in case:
        grid = _grid(case, mesh)
        axes = [torch.arange(m, device="cuda", dtype=torch.float64) * ((hi - lo) / (m - 1)) + lo
                for m, lo, hi in zip(grid.n, grid.lo, grid.hi)]
        z, y, x = torch.meshgrid(axes[2], axes[1], axes[0], indexing="ij")
        p = torch.stack([x.ravel(), y.ravel(), z.ravel()])
    else:
        p = _points(case if kind != "radius" else dict(n=n, where="near"), mesh, seed).to(dt)
    d, at = _exact_distances(p, mesh, dt, signed)
    if kind == "call_grid":
        return d
    if kind == "radius":
        r2 = float(case["reach"]) ** 2
        near = d * d <= r2
        at = torch.where(near[:, None], at, torch.zeros_like(at))
        return (None, torch.where(near, d * d, torch.full_like(d, r2)), at[:, 0], at[:, 1], at[:, 2])
    if kind == "call_points":
        return (d, at[:, 0], at[:, 1], at[:, 2], None) if case["output"] == "closest" else d
    return d, None
