"""GPU: edf_celllist on device arrays with the most triangles it takes, 2^26, which is one more than a mesh
handle takes. All but a few triangles are one far point, so the answer is that of the few."""

import numpy as np
import pytest
import torch

import oracle
import ssdf_b200 as S
from ssdf_b200 import workloads as W

pytestmark = pytest.mark.gpu


def arrays(nt):
    few = W.icosphere(1)
    at = torch.randperm(nt, generator=torch.Generator().manual_seed(1))[: few.nt].sort().values.cuda()
    s = []
    for k in range(3):
        c = torch.full((nt,), few.nv, dtype=torch.int32, device="cuda")
        c[at] = torch.tensor(few.triangles[:, k], dtype=torch.int32, device="cuda")
        s.append(c)
    return few, at.cpu().numpy(), s, np.concatenate([few.vertices, [[50.0, 60.0, 70.0]]])


def test_most_triangles():
    few, at, s, vertices = arrays(1 << 26)
    v = [torch.tensor(np.ascontiguousarray(a), dtype=torch.float32, device="cuda") for a in vertices.T]
    pts = np.random.default_rng(2).uniform(-1.5, 1.5, (3, 20)).astype(np.float32)
    p = [torch.tensor(np.ascontiguousarray(a), device="cuda") for a in pts]
    out = torch.full((20,), torch.finfo(torch.float32).max, dtype=torch.float32, device="cuda")
    tri = torch.full((20,), -1, dtype=torch.int32, device="cuda")
    S.edf_device(1, *p, *s, *v, out, tri)
    torch.cuda.synchronize()
    want, wtri = oracle.edf(pts, few, dtype=np.float32, with_index=True)
    assert np.array_equal(out.cpu().numpy(), want)
    assert np.array_equal(tri.cpu().numpy(), at[wtri])
    # a mesh handle still refuses that many
    with pytest.raises(RuntimeError, match="2\\^26"):
        S.DeviceMesh.from_device(*s, *v, keep_fp64=False, normals=False, treelet=0)
