"""GPU: the float arithmetic on meshes far from the origin, where the closest point's own rounding (of the
place, not of the mesh's size) decides between many triangles at nearly the same distance. Thousands of
overlapping triangles of size 1 face (1, 1, 1), the direction of their offset, in a slab about as thick as
that rounding; points lie in front of and behind them. Value and index equal the oracle's brute force in
float bit for bit, from float and from double vertices, in every walk."""

import numpy as np
import pytest
import torch

import oracle
import ssdf_b200 as S
from ssdf_b200 import workloads as W
from test_gpu_oriented_boxes import WALKS, run

pytestmark = pytest.mark.gpu

NORMAL = np.ones(3) / np.sqrt(3.0)


def slab(n, offset, thickness, seed):
    rng = np.random.default_rng(seed)
    a = np.array([1.0, -1.0, 0.0]) / np.sqrt(2.0)
    b = np.cross(NORMAL, a)
    centre = rng.uniform(-3, 3, (n, 2))
    corner = centre[:, None, :] + rng.uniform(-0.5, 0.5, (n, 3, 2))
    depth = thickness * rng.uniform(-1, 1, (n, 1, 1))
    v = offset + corner[..., :1] * a + corner[..., 1:] * b + depth * NORMAL
    return W.Mesh(v.reshape(-1, 3), np.arange(3 * n, dtype=np.int32).reshape(-1, 3))


def points(offset, n, seed):
    rng = np.random.default_rng(seed)
    a = np.array([1.0, -1.0, 0.0]) / np.sqrt(2.0)
    b = np.cross(NORMAL, a)
    away = rng.choice([-1.0, 1.0], (n, 1)) * 10.0 ** rng.uniform(1.0, 2.1, (n, 1))
    side = rng.uniform(-3, 3, (n, 2))
    return np.ascontiguousarray((offset + side[:, :1] * a + side[:, 1:] * b + away * NORMAL).T.astype(np.float32))


@pytest.mark.parametrize("walk", list(WALKS))
@pytest.mark.parametrize("doubles", [False, True])
@pytest.mark.parametrize("n, offset", [(2000, 16500.0), (20000, 16500.0), (20000, 4100.0)])
def test_float_winner_far_from_the_origin(n, offset, doubles, walk, monkeypatch):
    for k, v in WALKS[walk].items():
        monkeypatch.setenv(k, v)
    mesh = slab(n, offset, thickness=2.0 ** -23 * offset, seed=n)
    if not doubles:
        mesh = W.Mesh(mesh.vertices.astype(np.float32).astype(np.float64), mesh.triangles)
    pts = points(offset, 1500, seed=3)
    want, wtri = oracle.edf(pts, mesh, dtype=np.float32, with_index=True)
    dm = S.DeviceMesh(mesh, keep_fp64=True, normals=False) if doubles else \
        S.DeviceMesh(mesh, np.float32, keep_fp64=False, normals=False)
    got, tri = run(dm, pts, S.PREC_F32, torch.float32)
    dm.close()
    wrong = np.flatnonzero((got != want) | (tri != wtri))
    assert wrong.size == 0, (wrong.size, got[wrong[:5]], want[wrong[:5]])
