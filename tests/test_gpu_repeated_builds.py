"""GPU: a refined build is the same tree every time. The refinement's warps share subtrees that other warps
have just written; a read that ran ahead of one would give another tree, with another number of box and
triangle tests. The order in which warps arrive differs from build to build, the tree must not."""

import numpy as np
import pytest
import torch

import ssdf_b200 as S
from ssdf_b200 import capi
from ssdf_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nu, nv", [(24, 12), (160, 80), (400, 200)])
def test_refined_trees_do_not_depend_on_arrival_order(nu, nv, monkeypatch):
    mesh = W.torus(nu=nu, nv=nv, jitter=0.01)
    lo, hi = mesh.bbox()
    pts = np.random.default_rng(1).uniform(lo - 0.1, hi + 0.1, (4000, 3)).T
    x, y, z = (torch.tensor(np.ascontiguousarray(a), device="cuda") for a in pts)
    monkeypatch.setenv("SSDF_B200_COUNT", "1")
    monkeypatch.setenv("SSDF_B200_TRAVERSAL", "thread")
    seen = set()
    for _ in range(12):
        dm = S.DeviceMesh(mesh, treelet=3)
        out = torch.full((x.numel(),), torch.finfo(torch.float64).max, dtype=torch.float64, device="cuda")
        dm.query_points(x, y, z, out, None, precision=S.PREC_F64, output=S.OUT_EDF)
        counts = capi.last_query_counts()
        dm.close()
        seen.add((counts["triangle_tests"], counts["box_tests"], out.cpu().numpy().tobytes()))
    assert len(seen) == 1
