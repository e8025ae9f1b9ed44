"""GPU: meshes with NaN or infinite vertex coordinates among ordinary triangles. Such a triangle may have no
distance, or one by the corner that is finite; every walk must still answer as the oracle's brute force does,
bit for bit, whatever such triangles do to the boxes they share."""

import numpy as np
import pytest
import torch

import oracle
import ssdf_b200 as S
from ssdf_b200 import workloads as W
from test_gpu_oriented_boxes import WALKS, run

pytestmark = pytest.mark.gpu


def broken(kind, share, seed):
    mesh = W.random_soup(700, seed=seed)
    v = mesh.vertices.copy()
    rng = np.random.default_rng(seed)
    for t in rng.permutation(mesh.nt)[: max(1, int(share * mesh.nt))]:
        c = mesh.triangles[t]
        if kind == "nan corner":
            v[c[rng.integers(3)]] = np.nan
        elif kind == "nan triangle":
            v[c] = np.nan
        elif kind == "nan axis":
            v[c, rng.integers(3)] = np.nan
        elif kind == "inf corner":
            v[c[rng.integers(3)], rng.integers(3)] = rng.choice([-np.inf, np.inf])
        else:
            v[c] = rng.choice([-np.inf, np.inf], (3, 3))
    return W.Mesh(v, mesh.triangles)


@pytest.mark.parametrize("walk", list(WALKS))
@pytest.mark.parametrize("share", [0.0, 0.05, 0.5])
@pytest.mark.parametrize("kind", ["nan corner", "nan triangle", "nan axis", "inf corner", "inf triangle"])
def test_as_brute_force(kind, share, walk, monkeypatch):
    for k, v in WALKS[walk].items():
        monkeypatch.setenv(k, v)
    mesh = broken(kind, share, seed=11)
    pts = np.random.default_rng(12).uniform(-1.3, 1.3, (3, 500))
    dm = S.DeviceMesh(mesh, normals=False)
    want, wtri = oracle.edf(pts, mesh, with_index=True)
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
