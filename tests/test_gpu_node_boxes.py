"""GPU: node boxes built in blocks of 256 leaves, at sizes around one and two blocks, around runs of 32 in
the last block, and over many blocks. Distances and indices must equal the oracle's brute force bit for bit:
a box that misses one of its triangles loses it, and there is no tolerance."""

import numpy as np
import pytest
import torch

import oracle
import ssdf_b200 as S
from ssdf_b200 import workloads as W

pytestmark = pytest.mark.gpu


def soup(n, spread):
    """n small triangles: spread over a box, or with only 8 different centres (runs of equal Morton codes)."""
    rng = np.random.default_rng(n)
    c = rng.uniform(-1, 1, (n, 1, 3)) if spread else rng.uniform(-1, 1, (8, 1, 3))[rng.integers(0, 8, n)]
    v = (c + 0.03 * rng.normal(size=(n, 3, 3))).reshape(-1, 3)
    return W.Mesh(v, np.arange(3 * n, dtype=np.int32).reshape(n, 3))


@pytest.mark.parametrize("spread", [True, False])
@pytest.mark.parametrize("n", [5, 32, 255, 256, 257, 288, 511, 513, 543, 769, 6000])
def test_every_triangle_is_in_its_nodes(n, spread):
    mesh = soup(n, spread)
    v = mesh.vertices[mesh.triangles]
    pts = np.concatenate([v[:500].mean(1) + 0.001, np.random.default_rng(1).uniform(-1.3, 1.3, (300, 3))]).T.copy()
    want, wtri = oracle.edf(pts, mesh, with_index=True)
    x, y, z = (torch.tensor(a, device="cuda") for a in pts)
    dm = S.DeviceMesh(mesh)
    for prec in (S.PREC_F64, S.PREC_F32_FIXUP):
        out = torch.full((x.numel(),), torch.finfo(torch.float64).max, dtype=torch.float64, device="cuda")
        tri = torch.full((x.numel(),), -1, dtype=torch.int32, device="cuda")
        dm.query_points(x, y, z, out, tri, precision=prec, output=S.OUT_EDF)
        torch.cuda.synchronize()
        assert np.array_equal(out.cpu().numpy(), want) and np.array_equal(tri.cpu().numpy(), wtri), prec
    dm.close()
