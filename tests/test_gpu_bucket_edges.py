"""Counts and point-group witnesses over scenes at the edges of buckets (8
points) and level-1 nodes (32 buckets), at radii that reach little, half and
all of the scene, for a few queries and for packets."""
import numpy as np
import pytest

import rtdl_b200 as rt
from oracle import oracle as O
from rtdl_b200.runtime import pack_point_groups

pytestmark = pytest.mark.gpu


def _cols(rng, n, dim):
    p = rng.random((n, dim)).astype(np.float32).astype(np.float64)
    d = {"id": rng.permutation(n).astype(np.uint32), "x": p[:, 0], "y": p[:, 1]}
    if dim == 3:
        d["z"] = p[:, 2]
    return d


def _pack(c):
    return rt.pack_points(ids=c["id"], x=c["x"], y=c["y"], z=c.get("z"))


@pytest.mark.parametrize("nq", [3, 300])
@pytest.mark.parametrize("ns", [1, 7, 8, 9, 255, 256, 257, 8193])
def test_counts_and_witnesses(gpu, ns, nq):
    import torch

    rng = np.random.default_rng(100 * ns + nq)
    s2, q2, s3, q3 = _cols(rng, ns, 2), _cols(rng, nq, 2), _cols(rng, ns, 3), _cols(rng, nq, 3)
    half = ns // 2  # two groups, the second of them inside a smaller box than its points'
    groups = pack_point_groups([
        {"id": 0, "point_offset": 0, "point_count": half, "min_x": 0.0, "min_y": 0.0, "max_x": 1.0, "max_y": 1.0},
        {"id": 1, "point_offset": half, "point_count": ns - half, "min_x": 0.4, "min_y": 0.4, "max_x": 0.6,
         "max_y": 0.6}])
    out = [torch.zeros(nq, dtype=torch.int32, device="cuda") for _ in range(3)]
    for radius in (0.02, 0.5, 3.0):
        for threshold in (0, 4):
            exp = O.fixed_radius_count_threshold(q2, s2, radius=radius, threshold=threshold, threads=8)
            rows = rt.fixed_radius_count_threshold_2d(_pack(q2), _pack(s2), radius=radius, threshold=threshold)
            assert [r["neighbor_count"] for r in rows] == exp["neighbor_count"].tolist()
            assert [r["threshold_reached"] for r in rows] == exp["threshold_reached"].tolist()
        exp = O.fixed_radius_count_threshold(q3, s3, radius=radius, threshold=5, threads=8)
        with rt.prepare_b200_fixed_radius_count_threshold_3d(_pack(s3), max_radius=3.0) as prep:
            prep.write_device_count_threshold_columns(_pack(q3), radius=radius, threshold=5, query_ids_out=out[0],
                                                      neighbor_counts_out=out[1], threshold_flags_out=out[2])
        assert np.array_equal(out[1].cpu().numpy(), exp["neighbor_count"])
        assert np.array_equal(out[2].cpu().numpy(), exp["threshold_reached"])
        with rt.prepare_b200_point_group_nearest_witness_2d(_pack(s2), groups, max_radius=3.0) as prep:
            _, flags, rows, _ = O.point_group_witness(q2, s2, groups, radius=radius, threshold=3)
            assert np.array_equal(prep.threshold_flags(_pack(q2), radius=radius, threshold=3), flags)
            got = prep.nearest_witness_rows(_pack(q2), radius=radius)
            assert [r["neighbor_id"] for r in got] == rows["neighbor_id"].tolist()
            assert np.array_equal(np.array([r["distance"] for r in got]).view(np.uint64), rows["distance"].view(np.uint64))
