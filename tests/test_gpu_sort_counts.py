"""GPU: a sort tile that gives up on its predecessors' published counts counts their keys itself. Tiles wait
tens of thousands of polls, so that never happens by itself; here every tile counts for itself. Builds (30-bit
keys, 64-bit edge keys for the pseudo-normals) and point orders are the same."""

import numpy as np
import pytest
import torch

import ssdf_b200 as S
from ssdf_b200 import workloads as W

pytestmark = pytest.mark.gpu


def answers(mesh, pts):
    dm = S.DeviceMesh(mesh)
    x, y, z = (torch.tensor(a, device="cuda") for a in pts)
    out = torch.empty(x.numel(), dtype=torch.float64, device="cuda")
    tri = torch.empty(x.numel(), dtype=torch.int32, device="cuda")
    dm.query_points(x, y, z, out, tri, output=S.OUT_SDF)
    torch.cuda.synchronize()
    stats = dm.stats()
    dm.close()
    return out.cpu().numpy(), tri.cpu().numpy(), stats


@pytest.mark.parametrize("n", [2048, 2049, 4097, 26625, 100003])
def test_tiles_that_count_for_themselves(n, monkeypatch):
    nu = max(24, int(np.sqrt(n)))
    mesh = W.torus(nu=nu, nv=nu // 2, jitter=0.01)
    pts = np.random.default_rng(n).uniform(-1.5, 1.5, (n, 3)).T.copy()
    monkeypatch.setenv("SSDF_B200_WARP_POINTS", "0")
    want = answers(mesh, pts)
    monkeypatch.setenv("SSDF_B200_SORT_ALONE", "1")
    got = answers(mesh, pts)
    assert got[2] == want[2]
    assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1])
