"""GPU: mesh builds and point sorts at the sizes where their kernels change shape: sort tiles of 2,048 keys (one
short of a tile, whole tiles, one over), treelets from seven triangles on, warps that start from 16 or 32
triangles (below and above 100,000). A key lost or a subtree dropped changes an answer: distances and indices
must equal the oracle's brute force, and each other over tree shapes, bit for bit."""

import numpy as np
import pytest
import torch

import oracle
import ssdf_b200 as S
from ssdf_b200 import workloads as W

pytestmark = pytest.mark.gpu


def soup(n):
    rng = np.random.default_rng(n)
    v = (rng.uniform(-1, 1, (n, 1, 3)) + 0.02 * rng.normal(size=(n, 3, 3))).reshape(-1, 3)
    return W.Mesh(v, np.arange(3 * n, dtype=np.int32).reshape(n, 3))


def ask(dm, pts):
    x, y, z = (torch.tensor(a, device="cuda") for a in pts)
    out = torch.full((x.numel(),), torch.finfo(torch.float64).max, dtype=torch.float64, device="cuda")
    tri = torch.full((x.numel(),), -1, dtype=torch.int32, device="cuda")
    dm.query_points(x, y, z, out, tri, output=S.OUT_EDF)
    torch.cuda.synchronize()
    return out.cpu().numpy(), tri.cpu().numpy()


@pytest.mark.parametrize("n", [6, 7, 8, 17, 33, 2047, 2048, 2049, 4097, 100001])
def test_builds_with_and_without_treelets(n):
    mesh = soup(n)
    ids = np.random.default_rng(2).permutation(n)[:150]
    centres = mesh.vertices[mesh.triangles[ids]].mean(1) + 1e-3
    pts = np.concatenate([centres, np.random.default_rng(3).uniform(-1.2, 1.2, (100, 3))]).T.copy()
    want, wtri = oracle.edf(pts, mesh, with_index=True)
    for rounds in (0, 3):
        dm = S.DeviceMesh(mesh, treelet=rounds)
        got, tri = ask(dm, pts)
        dm.close()
        assert np.array_equal(got, want) and np.array_equal(tri, wtri), rounds


@pytest.mark.parametrize("n", [26623, 26624, 26625])
def test_point_sorts_around_whole_tiles(n):
    """Every point of a sorted list gets its own answer: equal to the same points asked in short lists."""
    mesh = W.torus(nu=30, nv=15, jitter=0.02)
    pts = np.random.default_rng(n).uniform(-1.5, 1.5, (n, 3)).T.copy()
    dm = S.DeviceMesh(mesh)
    got, tri = ask(dm, pts)
    half = [ask(dm, pts[:, k].copy()) for k in (slice(0, 13000), slice(13000, 20000), slice(20000, n))]
    dm.close()
    assert np.array_equal(got, np.concatenate([h[0] for h in half]))
    assert np.array_equal(tri, np.concatenate([h[1] for h in half]))
