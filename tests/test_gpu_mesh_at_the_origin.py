"""GPU: a mesh whose triangles are all one point at the origin or next to it, queried there and elsewhere. All
distances tie, the square of any share of the coordinates' magnitude is zero, and the answer is the lowest index in
every arithmetic and walk."""

import numpy as np
import pytest
import torch

import oracle
import ssdf_b200 as S
from ssdf_b200 import workloads as W
from test_gpu_oriented_boxes import WALKS, run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("walk", list(WALKS))
@pytest.mark.parametrize("place", [0.0, 1e-25])
@pytest.mark.parametrize("nt", [3, 300, 5000])
def test_ties_at_the_origin(nt, place, walk, monkeypatch):
    for k, v in WALKS[walk].items():
        monkeypatch.setenv(k, v)
    mesh = W.Mesh(np.full((3, 3), place), np.tile(np.arange(3, dtype=np.int32), (nt, 1)))
    pts = np.array([[place] * 3, [0.0, 0.0, 0.0], [1e-30, 0.0, 0.0], [1e-20, 1e-25, 0.0], [0.3, -0.2, 0.1]]).T.copy()
    want, wtri = oracle.edf(pts, mesh, with_index=True)
    assert np.all(wtri == 0)
    dm = S.DeviceMesh(mesh, normals=False)
    for prec in (S.PREC_F64, S.PREC_F32_FIXUP):
        got, tri = run(dm, pts, prec, torch.float64)
        assert np.array_equal(got, want) and np.array_equal(tri, wtri), prec
    dm.close()
    single = S.DeviceMesh(mesh, np.float32, keep_fp64=False, normals=False)
    want, wtri = oracle.edf(pts.astype(np.float32), mesh, dtype=np.float32, with_index=True)
    got, tri = run(single, pts.astype(np.float32), S.PREC_F32, torch.float32)
    single.close()
    assert np.array_equal(got, want) and np.array_equal(tri, wtri)
