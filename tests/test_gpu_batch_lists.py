"""GPU: the hand-over lists of batches in the plain arithmetics are a help, not a need. Reserving for any number
of queries succeeds, a job too large for a launch of its own to keep a list keeps none in a batch either, and
jobs with and without one give the same bits as their launches alone."""

import numpy as np
import pytest
import torch

import ssdf_b200 as S
from ssdf_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [S.PREC_F64, S.PREC_F32])
def test_reserving_for_more_than_the_memory_holds(precision):
    b = S.Batch(4, precision)
    b.reserve(1 << 40)
    b.close()


def grid_job(mesh, n):
    dm = S.DeviceMesh(mesh)
    grid = W.Grid.padded_nodes(mesh, n, 0.2)
    outs = [torch.empty(grid.size, dtype=torch.float64, device="cuda") for _ in range(2)]
    return dm, grid, outs


@pytest.mark.parametrize("precision", [S.PREC_F64, S.PREC_F32_FIXUP])
def test_large_plain_job_keeps_no_list(precision):
    """261^3 nodes (above 2^24) in double, in a fix-up batch on a mesh of needles, beside a small job."""
    jobs = [grid_job(W.beam_lattice(40), 261), grid_job(W.icosphere(3), 24)]
    big = jobs[0][1].size
    assert big > 1 << 24
    for dm, grid, outs in jobs:
        dm.query_grid(grid, outs[0], None, precision=S.PREC_F64, output=S.OUT_SDF)
    b = S.Batch(4, precision)
    for dm, grid, outs in jobs:
        b.add_grid(dm, grid, outs[1], None)
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    b.run(use_graph=False)
    torch.cuda.synchronize()
    held = before - torch.cuda.mem_get_info()[0]
    assert held < 4 * big, held  # a list would hold 8 bytes a query
    for _, _, (alone, batched) in jobs:
        assert torch.equal(alone, batched)
    b.close()
    for dm, _, _ in jobs:
        dm.close()
