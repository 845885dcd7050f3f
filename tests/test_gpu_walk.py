"""Sizes at which the tree walks, the packets and the sorts change shape:
bucket and level edges of the search tree (8 points a bucket, 32 nodes a
level), the query counts at which packets narrow, the list sizes of the KNN
paths, dense and sparse packets, and the tile edges of the radix sort.  Rows
must be the oracle's bit for bit (ids, exact FP64 distances, order).
"""
import numpy as np
import pytest

import rtdl_b200 as rt
from oracle import oracle as O
from rtdl_b200.batch import B200ProblemBatch

pytestmark = pytest.mark.gpu


def _cols(pts, ids=None):
    ids = np.arange(len(pts), dtype=np.uint32) if ids is None else ids
    d = {"id": ids, "x": pts[:, 0], "y": pts[:, 1]}
    if pts.shape[1] == 3:
        d["z"] = pts[:, 2]
    return d


def _pack(c):
    return rt.pack_points(ids=c["id"], x=c["x"], y=c["y"], z=c.get("z"))


def _same(view, exp, ranked):
    got = view.to_numpy()
    assert len(got) == len(exp)
    for f in ("query_id", "neighbor_id") + (("neighbor_rank",) if ranked else ()):
        assert np.array_equal(got[f], exp[f]), f
    assert np.array_equal(got["distance"].view(np.uint64), exp["distance"].view(np.uint64))
    view.close()


def _uneven(rng, n, dim):
    """Half in a few tight clumps (with repeated points), half spread out, FP32 values."""
    pts = rng.random((n, dim))
    half = n // 2
    pts[:half] = rng.random((4, dim))[rng.integers(0, 4, half)] + rng.normal(0.0, 0.004, (half, dim))
    pts[: half // 8] = pts[half // 8: 2 * (half // 8)]
    return rng.permutation(pts).astype(np.float32).astype(np.float64)


@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("n", [1, 7, 8, 9, 255, 256, 257, 8191, 8192, 8193])
def test_tree_edges(gpu, n, dim):
    rng = np.random.default_rng(1000 * dim + n)
    s, q = _cols(_uneven(rng, n, dim)), _cols(_uneven(rng, 97, dim))
    with rt.B200Scene(_pack(s)) as scene:
        for radius, k in ((0.02, 64), (0.3, 3), (4.0, 64)):
            v = scene.query(_pack(q), predicate="fixed_radius_neighbors", radius=radius, limit=k)
            _same(v, O.fixed_radius_neighbors(q, s, radius=radius, k_max=k, threads=8), False)
        _same(scene.query(_pack(q), predicate="knn_rows", limit=9), O.knn_rows(q, s, k=9, threads=8), True)
        _, nd, ni = scene.directed_hausdorff(_pack(q), with_nearest=True)
    dist, nid = O.nearest(q, s, threads=8)
    assert np.array_equal(nd.view(np.uint64), dist.view(np.uint64)) and np.array_equal(ni, nid)


# the counts at which a packet's width goes from single queries to 8, 16 and 32, and a ragged last packet
@pytest.mark.parametrize("nq", [33, 4736, 4737, 56832, 56833, 113664, 113697])
def test_packet_widths(gpu, nq):
    rng = np.random.default_rng(nq)
    s, q = _cols(_uneven(rng, 20000, 3)), _cols(_uneven(rng, nq, 3))
    with rt.B200Scene(_pack(s)) as scene:
        for radius, k in ((0.003, 64), (0.04, 8)):  # the larger one: hundreds in radius inside a clump, cut to 8
            v, overflow = scene.query(_pack(q), predicate="fixed_radius_neighbors", radius=radius, limit=k,
                                      with_overflow=True)
            exp, counts = O.fixed_radius_neighbors(q, s, radius=radius, k_max=k, threads=8, with_counts=True)
            _same(v, exp, False)
            assert np.array_equal(overflow.astype(bool), counts > k)


@pytest.mark.parametrize("ns", [5, 63, 20000])
@pytest.mark.parametrize("k", [1, 8, 9, 16, 17, 32, 33, 64, 65])
def test_knn_list_sizes(gpu, k, ns):
    rng = np.random.default_rng(100 * k + ns)
    s = _cols(_uneven(rng, ns, 3))
    for nq in (50, 5000):  # one query a warp; packets
        q = _cols(_uneven(rng, nq, 3))
        with rt.B200Scene(_pack(s)) as scene:
            _same(scene.query(_pack(q), predicate="knn_rows", limit=k), O.knn_rows(q, s, k=k, threads=8), True)


@pytest.mark.parametrize("nq", [40, 5000])
def test_crowded_radius(gpu, nq):
    """Far more points in the radius than a query's list holds, many of them tied."""
    rng = np.random.default_rng(nq)
    s = _cols(np.round(rng.random((9000, 2)) * 24) / 256)
    q = _cols(np.round(rng.random((nq, 2)) * 24) / 256)
    with rt.B200Scene(_pack(s)) as scene:
        for radius, k in ((0.05, 64), (0.2, 1)):
            v = scene.query(_pack(q), predicate="fixed_radius_neighbors", radius=radius, limit=k)
            _same(v, O.fixed_radius_neighbors(q, s, radius=radius, k_max=k, threads=8), False)
        _same(scene.query(_pack(q), predicate="knn_rows", limit=32), O.knn_rows(q, s, k=32, threads=8), True)


@pytest.mark.parametrize("n", [1, 31, 4095, 4096, 4097, 8192, 12289])
def test_sort_tiles(gpu, n):
    """Search and query codes and unsorted query ids through one block, one tile and more."""
    rng = np.random.default_rng(n)
    s = _cols(_uneven(rng, n, 2))
    q = _cols(_uneven(rng, n, 2), ids=rng.integers(0, 1 << 32, n, dtype=np.uint64).astype(np.uint32))
    v = rt.runtime.fixed_radius_neighbors(_pack(q), _pack(s), radius=0.01, k_max=4)
    _same(v, O.fixed_radius_neighbors(q, s, radius=0.01, k_max=4, threads=8), False)


def test_sort_of_one_digit_by_problem(gpu):
    """Unsorted ids in a batch: the sort by problem takes a single pass (an odd number)."""
    rng = np.random.default_rng(3)
    sizes = (4097, 1, 700)
    rec = [rt.pack_points(**{("ids" if k == "id" else k): v for k, v in _cols(_uneven(rng, n, 3), ids=rng.permutation(n)
                                                                             .astype(np.uint32)).items()}).records
           for n in sizes + sizes]
    probes, builds = rec[:3], rec[3:]
    with B200ProblemBatch(builds) as batch:
        out = batch.fixed_radius_neighbors(probes, radius=[0.01, 2.0, 0.02], k_max=64)
    for p in range(3):
        exp = O.fixed_radius_neighbors(probes[p], builds[p], radius=[0.01, 2.0, 0.02][p], k_max=64)
        got = out.problem(p)
        assert np.array_equal(got["query_id"], exp["query_id"])
        assert np.array_equal(got["neighbor_id"], exp["neighbor_id"])
        assert np.array_equal(got["distance"].view(np.uint64), exp["distance"].view(np.uint64))
