"""GPU: walks cull at every scale of a mesh that the arithmetic has distances for. The boxes' frame is scaled
by a power of two where the mesh is very large or very small; answers equal the oracle's brute force bit for
bit, and a query tests less than a tenth of the triangles on average (without culling, all of them)."""

import numpy as np
import pytest
import torch

import oracle
import ssdf_b200 as S
from ssdf_b200 import capi
from ssdf_b200 import workloads as W
from test_gpu_oriented_boxes import WALKS, moved, run

pytestmark = pytest.mark.gpu

TORUS = W.torus(nu=100, nv=50, jitter=0.01)


def near(mesh, n, seed):
    rng = np.random.default_rng(seed)
    lo, hi = mesh.bbox()
    size = (hi - lo).max()
    c = mesh.vertices[mesh.triangles[rng.integers(0, mesh.nt, n)]].mean(1)
    return np.ascontiguousarray((c + 0.02 * size * rng.normal(size=(n, 3))).T)


def ask(dm, pts, precision, dtype, monkeypatch):
    monkeypatch.setenv("SSDF_B200_COUNT", "1")
    got, tri = run(dm, pts, precision, dtype)
    tests = capi.last_query_counts()["triangle_tests"] / pts.shape[1]
    monkeypatch.delenv("SSDF_B200_COUNT")
    return got, tri, tests


# packets test the triangles that any of 32 unsorted points wants, so their counts say nothing here
@pytest.mark.parametrize("walk", ["warp", "thread", "packet, handed over"])
@pytest.mark.parametrize("scale", [1e-100, 1e-42, 1e-30, 1e-19, 1e-10, 1e9, 1e15, 1e19, 1e32, 1e37])
def test_double(scale, walk, monkeypatch):
    for k, v in WALKS[walk].items():
        monkeypatch.setenv(k, v)
    mesh = moved(TORUS, scale)
    pts = near(mesh, 1500, seed=1)
    want, wtri = oracle.edf(pts, mesh, with_index=True)
    dm = S.DeviceMesh(mesh, normals=False)
    for prec in (S.PREC_F64, S.PREC_F32_FIXUP):
        got, tri, tests = ask(dm, pts, prec, torch.float64, monkeypatch)
        assert np.array_equal(got, want) and np.array_equal(tri, wtri), prec
        assert walk == "packet, handed over" or tests < mesh.nt / 10, (prec, tests)
    dm.close()


@pytest.mark.parametrize("walk", ["warp", "thread", "packet, handed over"])
@pytest.mark.parametrize("scale", [1e-42, 1e-24, 1e-15, 1e-10, 1e9, 1e15, 1e17, 1e25])
def test_float(scale, walk, monkeypatch):
    for k, v in WALKS[walk].items():
        monkeypatch.setenv(k, v)
    mesh = moved(TORUS, scale)
    mesh = W.Mesh(mesh.vertices.astype(np.float32).astype(np.float64), mesh.triangles)
    pts = near(mesh, 1500, seed=2).astype(np.float32)
    want, wtri = oracle.edf(pts, mesh, dtype=np.float32, with_index=True)
    dm = S.DeviceMesh(mesh, np.float32, keep_fp64=False, normals=False)
    got, tri, tests = ask(dm, pts, S.PREC_F32, torch.float32, monkeypatch)
    dm.close()
    assert np.array_equal(got, want) and np.array_equal(tri, wtri)
    # below 1e-15 the squares are at or below float's smallest normal number: ties, all of them to be met
    assert scale < 1e-15 or walk == "packet, handed over" or tests < mesh.nt / 10, tests


def test_collapsed_mesh_of_tiny_extent():
    """Triangles that are points, closer together than the frame is left unscaled for: the fix-up path."""
    rng = np.random.default_rng(7)
    mesh = W.Mesh(1e-12 * rng.uniform(-1, 1, (600, 3)), np.repeat(np.arange(600, dtype=np.int32), 3).reshape(-1, 3))
    pts = np.ascontiguousarray(1e-12 * rng.uniform(-1.5, 1.5, (3, 400)))
    want, wtri = oracle.edf(pts, mesh, with_index=True)
    dm = S.DeviceMesh(mesh, normals=False)
    for prec in (S.PREC_F64, S.PREC_F32_FIXUP):
        got, tri = run(dm, pts, prec, torch.float64)
        assert np.array_equal(got, want) and np.array_equal(tri, wtri), prec
    dm.close()


def test_points_whose_distance_overflows_are_not_walked(monkeypatch):
    mesh = TORUS
    pts = np.array([[1e160, 0.0, 0.0], [0.0, -1e200, 1.0], [1e300, 1e300, 1e300]]).T.copy()
    dm = S.DeviceMesh(mesh, normals=False)
    got, tri, tests = ask(dm, pts, S.PREC_F64, torch.float64, monkeypatch)
    dm.close()
    assert np.all(np.isinf(got) | (got == np.finfo(np.float64).max)) and np.all(tri == -1) and tests == 0
