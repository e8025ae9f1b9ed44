"""GPU: point lists in Morton order, as packets, against input order, for lists that a warp a query would
otherwise answer (SSDF_B200_WARP_POINTS=0 takes that walk away from both sides): every output kind, lists
around the length from which they are sorted, points that keep their incoming bound. Bit for bit equal, and
equal to the oracle on a sample."""

import numpy as np
import pytest

import oracle
import ssdf_b200 as S
from ssdf_b200 import capi
from ssdf_b200 import workloads as W
from test_gpu_sorted_points import _points

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def no_warp_walk(monkeypatch):
    monkeypatch.setenv("SSDF_B200_WARP_POINTS", "0")


def both_orders(call, monkeypatch):
    monkeypatch.setenv("SSDF_B200_SORT_POINTS", "0")
    a = call()
    monkeypatch.setenv("SSDF_B200_SORT_POINTS", "1")
    return a, call()


@pytest.mark.parametrize("n", [4096, 4097, 9000])
@pytest.mark.parametrize("prec", ["f32x", "f64"])
def test_distances_in_both_orders(n, prec, monkeypatch):
    mesh = W.torus_knot_tube(nu=192, nv=24)
    pts = _points(mesh, n, seed=n)
    monkeypatch.setenv("SSDF_B200_PRECISION", prec)
    (d0, t0), (d1, t1) = both_orders(lambda: S.edf_index(pts, mesh), monkeypatch)
    assert np.array_equal(d0, d1) and np.array_equal(t0, t1)
    (s0, i0), (s1, i1) = both_orders(lambda: S.sdf_points(pts, mesh), monkeypatch)
    assert np.array_equal(s0, s1) and np.array_equal(i0, i1)
    ids = np.arange(0, n, 97)
    want, wtri = oracle.edf(pts[:, ids].copy(), mesh, with_index=True)
    assert np.array_equal(d1[ids], want) and np.array_equal(t1[ids], wtri)


@pytest.mark.parametrize("n", [4096, 9000])
def test_closest_points_and_incoming_bounds_in_both_orders(n, monkeypatch):
    mesh = W.icosphere(3)
    pts = _points(mesh, n, seed=4)
    init = np.where(np.arange(n) % 3 == 0, 0.01, np.finfo(np.float64).max)
    a, b = both_orders(lambda: S.closest_point_bvh(pts, mesh, outd=init), monkeypatch)
    for x, y, name in zip(a, b, ("d", "x", "y", "z", "tri")):
        assert np.array_equal(x, y), name
    kept = b[0] == init
    assert kept.any() and not kept.all()


def test_the_orders_are_walked_differently(monkeypatch):
    """What the comparisons rest on: a sorted list walks as packets, whose lanes test each other's triangles."""
    mesh = W.icosphere(4)
    pts = _points(mesh, 4096, seed=1)
    monkeypatch.setenv("SSDF_B200_COUNT", "1")
    monkeypatch.setenv("SSDF_B200_WARP_BUDGET", "0")

    def tests():
        S.edf_index(pts, mesh)
        return capi.last_query_counts()["box_tests"]

    a, b = both_orders(tests, monkeypatch)
    assert a != b
