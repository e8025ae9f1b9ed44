"""GPU: the oriented boxes the query kernels walk, at the edges of their construction and of their
margins. Every arithmetic must equal the oracle's brute force bit for bit (distance and index; the box
walk only skips triangles, so there is no tolerance):
  - mesh sizes around the leaf size and around the largest subtree that gets oriented boxes (64);
  - slivers below and above the aspect ratio from which a child keeps its axis-aligned box;
  - scales and offsets at which the box frame is moved, scaled, or culls nothing;
  - collinear and collapsed triangles, planar meshes (a zero half extent), points far away, NaN, inf."""

import numpy as np
import pytest
import torch

import oracle
import ssdf_b200 as S
from ssdf_b200 import workloads as W

pytestmark = pytest.mark.gpu


def slivers(n, aspect, seed=0):
    rng = np.random.default_rng(seed)
    a = rng.uniform(-1, 1, (n, 3))
    u, w = rng.normal(size=(n, 3)), rng.normal(size=(n, 3))
    u /= np.linalg.norm(u, axis=1, keepdims=True)
    w -= (w * u).sum(1, keepdims=True) * u
    w /= np.linalg.norm(w, axis=1, keepdims=True)
    length = rng.uniform(0.1, 0.5, (n, 1))
    v = np.stack([a, a + length * u, a + 0.4 * length * u + length / aspect * w], 1).reshape(-1, 3)
    return W.Mesh(v, np.arange(3 * n, dtype=np.int32).reshape(-1, 3))


def sheet(n):
    """A planar, axis-aligned sheet of 2 n^2 triangles."""
    g = np.linspace(0.0, 1.0, n + 1)
    v = np.stack(np.meshgrid(g, g, [0.25], indexing="ij"), -1).reshape(-1, 3)
    i, j = np.meshgrid(np.arange(n), np.arange(n), indexing="ij")
    a = (i * (n + 1) + j).ravel()
    t = np.concatenate([np.stack([a, a + 1, a + n + 2], 1), np.stack([a, a + n + 2, a + n + 1], 1)])
    return W.Mesh(v, t.astype(np.int32))


def collapsed():
    m = W.random_soup(90, seed=8)
    t = m.triangles.copy()
    t[::3, 2] = t[::3, 1]
    t[::9, 1] = t[::9, 2] = t[::9, 0]
    return W.Mesh(m.vertices, t)


def moved(mesh, scale, offset=0.0):
    return W.Mesh(mesh.vertices * scale + offset, mesh.triangles)


MESHES = {
    **{f"soup{n}": W.random_soup(n, seed=n) for n in (1, 2, 4, 5, 63, 64, 65, 66, 130)},
    "torus": W.torus(nu=40, nv=20, jitter=0.01),
    "sheet": sheet(17),
    "collapsed": collapsed(),
    **{f"aspect{a}": slivers(300, a) for a in (30, 1500, 2500, 1e5)},
    "beams": W.beam_lattice(60),
    "offset 25000": moved(W.torus(nu=40, nv=20, jitter=0.01), 1.0, 25000.0),
    "offset 1e6": moved(W.icosphere(2), 1.0, 1e6),
    "scale 1e-9": moved(W.torus(nu=40, nv=20, jitter=0.01), 1e-9),
    "scale 1e-24": moved(W.icosphere(2), 1e-24),
    "scale 1e19": moved(W.icosphere(2), 1e19),
    "scale 1e25": moved(W.icosphere(2), 1e25),
}


def queries(mesh):
    rng = np.random.default_rng(5)
    lo, hi = mesh.bbox()
    size = (hi - lo).max()
    v = mesh.vertices[mesh.triangles]
    near = v.mean(1)[rng.integers(0, mesh.nt, 300)] + 0.02 * size * rng.normal(size=(300, 3))
    box = rng.uniform(lo - 0.3 * size, hi + 0.3 * size, (300, 3))
    far = mesh.vertices.mean(0) + size * rng.normal(size=(30, 3)) * 10.0 ** rng.uniform(0, 6, (30, 1))
    return np.concatenate([near, box, far, mesh.vertices[:40], v.mean(1)[:40]]).T.copy()


def run(dm, pts, precision, dtype):
    x, y, z = (torch.tensor(a, dtype=dtype, device="cuda") for a in pts)
    out = torch.full((x.numel(),), torch.finfo(dtype).max, dtype=dtype, device="cuda")
    tri = torch.full((x.numel(),), -1, dtype=torch.int32, device="cuda")
    code = S.F64 if dtype == torch.float64 else S.F32
    dm.query_points(x, y, z, out, tri, precision=precision, output=S.OUT_EDF, coord_type=code, out_type=code)
    torch.cuda.synchronize()
    return out.cpu().numpy(), tri.cpu().numpy()


# a warp per query (short lists' default, and with a stack that sends lanes into their own subtrees), a
# thread per query, 32-query packets, packets that hand their queries to the second stage
WALKS = {"warp": {}, "warp, short stack": {"SSDF_B200_WINDOW_STACK": "3"}, "thread": {"SSDF_B200_WARP_POINTS": "0"},
         "packet": {"SSDF_B200_TRAVERSAL": "warp"},
         "packet, handed over": {"SSDF_B200_TRAVERSAL": "warp", "SSDF_B200_WARP_BUDGET": "2"}}


@pytest.mark.parametrize("walk", list(WALKS))
@pytest.mark.parametrize("name", list(MESHES))
def test_every_arithmetic_equals_brute_force(name, walk, monkeypatch):
    for k, v in WALKS[walk].items():
        monkeypatch.setenv(k, v)
    mesh = MESHES[name]
    pts = queries(mesh)
    want, wtri = oracle.edf(pts, mesh, with_index=True)
    dm = S.DeviceMesh(mesh)
    for prec in (S.PREC_F64, S.PREC_F32_FIXUP):
        got, tri = run(dm, pts, prec, torch.float64)
        assert np.array_equal(got, want) and np.array_equal(tri, wtri), prec
    dm.close()
    single = S.DeviceMesh(mesh, np.float32, keep_fp64=False, normals=False)
    p32 = pts.astype(np.float32)
    want, wtri = oracle.edf(p32, mesh, dtype=np.float32, with_index=True)
    got, tri = run(single, p32, S.PREC_F32, torch.float32)
    single.close()
    assert np.array_equal(got, want) and np.array_equal(tri, wtri)


@pytest.mark.parametrize("n", [1, 3, 4, 5, 24576, 24577])
def test_list_lengths_at_the_warp_walk_limit(n):
    """Both sides of the length up to which a warp answers each query, and partial blocks: equal to the
    oracle on a sample, and to the plain double kernel at every point."""
    mesh = W.torus(nu=30, nv=15, jitter=0.02)
    lo, hi = mesh.bbox()
    pts = np.random.default_rng(n).uniform(lo - 0.2, hi + 0.2, (n, 3)).T.copy()
    dm = S.DeviceMesh(mesh)
    got, tri = run(dm, pts, S.PREC_F32_FIXUP, torch.float64)
    d64, t64 = run(dm, pts, S.PREC_F64, torch.float64)
    dm.close()
    ids = np.arange(0, n, max(1, n // 500))
    want, wtri = oracle.edf(pts[:, ids].copy(), mesh, with_index=True)
    assert np.array_equal(got, d64) and np.array_equal(tri, t64)
    assert np.array_equal(got[ids], want) and np.array_equal(tri[ids], wtri)


def test_points_that_are_not_finite_keep_their_bound():
    mesh = MESHES["torus"]
    bad = [np.nan, np.inf, -np.inf]
    pts = np.array([[b if k == d else 0.1 for k in range(3)] for b in bad for d in range(3)]).T.copy()
    dm = S.DeviceMesh(mesh)
    for prec in (S.PREC_F64, S.PREC_F32_FIXUP):
        x, y, z = (torch.tensor(a, device="cuda") for a in pts)
        out = torch.full((9,), 3.5, dtype=torch.float64, device="cuda")
        tri = torch.full((9,), -7, dtype=torch.int32, device="cuda")
        dm.query_points(x, y, z, out, tri, precision=prec, output=S.OUT_EDF)
        torch.cuda.synchronize()
        assert np.all(out.cpu().numpy() == 3.5) and np.all(tri.cpu().numpy() == -7), prec
    dm.close()
