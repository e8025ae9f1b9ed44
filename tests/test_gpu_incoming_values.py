"""GPU: incoming squared distances that no distance meets (NaN, negative, zero) beside ordinary ones in the same
packets. Such a query keeps its value, and the others' answers are those they get without it, in every
arithmetic and walk."""

import numpy as np
import pytest
import torch

import ssdf_b200 as S
from ssdf_b200 import workloads as W
from test_gpu_oriented_boxes import WALKS

pytestmark = pytest.mark.gpu

MESH = W.torus(nu=60, nv=30, jitter=0.01)
PRECISIONS = {"f64": (S.PREC_F64, torch.float64), "f32x": (S.PREC_F32_FIXUP, torch.float64),
              "f32": (S.PREC_F32, torch.float32)}


def query(dm, points, grid, init, prec, dtype):
    code = S.F64 if dtype == torch.float64 else S.F32
    out = torch.tensor(init, dtype=dtype, device="cuda")
    if grid is not None:
        dm.query_grid(grid, out, None, precision=prec, output=S.OUT_SQEDF, coord_type=code, out_type=code)
    else:
        x, y, z = (torch.tensor(np.ascontiguousarray(a), dtype=dtype, device="cuda") for a in points)
        dm.query_points(x, y, z, out, None, precision=prec, output=S.OUT_SQEDF, coord_type=code, out_type=code)
    torch.cuda.synchronize()
    return out.cpu().numpy()


@pytest.mark.parametrize("precision", list(PRECISIONS))
@pytest.mark.parametrize("walk", [*WALKS, "grid"])
def test_values_that_no_distance_meets(walk, precision, monkeypatch):
    prec, dtype = PRECISIONS[precision]
    lo, hi = MESH.bbox()
    grid = W.Grid.padded_nodes(MESH, 24, 0.3) if walk == "grid" else None
    n = grid.size if grid else 8000
    rng = np.random.default_rng(3)
    points = None if grid else rng.uniform(lo - 0.3, hi + 0.3, (n, 3)).T
    dm = S.DeviceMesh(MESH)
    big = np.finfo(np.float64 if dtype == torch.float64 else np.float32).max
    plain = query(dm, points, grid, np.full(n, big), prec, dtype)
    init = np.full(n, big)
    kind = rng.integers(0, 12, n)
    for k, v in enumerate((np.nan, -1.0, -np.inf, 0.0, -0.0, 1e-3)):
        init[kind == k] = v
    for k, v in WALKS.get(walk, {}).items():
        monkeypatch.setenv(k, v)
    got = query(dm, points, grid, init, prec, dtype)
    dm.close()
    init = init.astype(got.dtype)
    want = np.where(plain < init, plain, init)
    assert np.array_equal(got, want, equal_nan=True), np.flatnonzero(~((got == want) | np.isnan(want)))[:5]
