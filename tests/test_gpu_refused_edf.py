"""GPU: a call over device arrays with a vertex index out of range is refused and leaves its in/out arrays as
they were, whichever way its size would have taken (every pair by warps or by tiles, the tree)."""

import numpy as np
import pytest
import torch

import ssdf_b200 as S
from ssdf_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("method", [0, 1])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("n, sub, bad", [(500, 1, 80), (500, 1, -1), (12000, 2, 200), (40000, 4, 1 << 20)])
def test_refused_call_writes_nothing(n, sub, bad, dtype, method):
    mesh = W.icosphere(sub)
    s = [torch.tensor(np.ascontiguousarray(a), dtype=torch.int32, device="cuda") for a in mesh.triangles.T]
    s[1][mesh.nt // 2] = bad
    assert bad < 0 or bad >= mesh.nv
    v = [torch.tensor(np.ascontiguousarray(a), dtype=dtype, device="cuda") for a in mesh.vertices.T]
    p = [torch.tensor(a, dtype=dtype, device="cuda") for a in np.random.default_rng(n).uniform(-1.5, 1.5, (3, n))]
    out = torch.full((n,), 3.5, dtype=dtype, device="cuda")
    tri = torch.full((n,), -7, dtype=torch.int32, device="cuda")
    with pytest.raises(RuntimeError, match="INVALID_ARGUMENT: triangle [0-9]+ has a vertex index"):
        S.edf_device(method, *p, *s, *v, out, tri)
    assert torch.all(out == 3.5) and torch.all(tri == -7)
