"""Points on the radius and within FP32 rounding of it, many to a bucket: which
of them count is decided in FP64, on the packet and the single-query paths, for
rows, counts and point groups, near the origin and far from it (where the FP32
error exceeds the points' spacing).
"""
import numpy as np
import pytest

import rtdl_b200 as rt
from oracle import oracle as O
from rtdl_b200.runtime import pack_point_groups

pytestmark = pytest.mark.gpu


def _cols(p):
    d = {"id": np.arange(len(p), dtype=np.uint32), "x": p[:, 0], "y": p[:, 1]}
    if p.shape[1] == 3:
        d["z"] = p[:, 2]
    return d


def _pack(c):
    return rt.pack_points(ids=c["id"], x=c["x"], y=c["y"], z=c.get("z"))


def _check(q, s, radius):
    exp, counts = O.fixed_radius_neighbors(q, s, radius=radius, k_max=64, threads=8, with_counts=True)
    with rt.B200Scene(_pack(s)) as scene:
        view, overflow = scene.query(_pack(q), predicate="fixed_radius_neighbors", radius=radius, limit=64,
                                     with_overflow=True)
        got = view.to_numpy()
        assert len(got) == len(exp)
        for f in ("query_id", "neighbor_id"):
            assert np.array_equal(got[f], exp[f]), f
        assert np.array_equal(got["distance"].view(np.uint64), exp["distance"].view(np.uint64))
        assert np.array_equal(overflow.astype(bool), counts > 64)
        view.close()
    if "z" not in s:
        rows = rt.fixed_radius_count_threshold_2d(_pack(q), _pack(s), radius=radius, threshold=0)
        assert np.array_equal(np.array([r["neighbor_count"] for r in rows]), counts)
        groups = pack_point_groups([{"id": 0, "point_offset": 0, "point_count": len(s["id"]), "min_x": s["x"].min(),
                                     "min_y": s["y"].min(), "max_x": s["x"].max(), "max_y": s["y"].max()}])
        with rt.prepare_b200_point_group_nearest_witness_2d(_pack(s), groups, max_radius=radius) as prep:
            for threshold in (1, 9):
                assert prep.count_threshold_reached(_pack(q), radius=radius, threshold=threshold) == \
                    int((counts >= threshold).sum())
    else:
        import torch

        out = [torch.zeros(len(counts), dtype=torch.int32, device="cuda") for _ in range(3)]
        with rt.prepare_b200_fixed_radius_count_threshold_3d(_pack(s), max_radius=radius) as prep:
            prep.write_device_count_threshold_columns(_pack(q), radius=radius, threshold=500, query_ids_out=out[0],
                                                      neighbor_counts_out=out[1], threshold_flags_out=out[2])
        assert np.array_equal(out[1].cpu().numpy(), np.minimum(counts, 500))


@pytest.mark.parametrize("offset", [0.0, 300.0])
@pytest.mark.parametrize("step", [1 / 64, 0.1])  # exact in FP32 and FP64; exact in neither
@pytest.mark.parametrize("dim,side", [(2, 120), (3, 24)])
@pytest.mark.parametrize("nq", [60, 6000])
def test_lattice(gpu, nq, dim, side, step, offset):
    rng = np.random.default_rng(side)
    grid = np.stack(np.meshgrid(*[np.arange(side)] * dim), -1).reshape(-1, dim).astype(np.float64)
    q = grid[rng.integers(0, len(grid), nq)]
    for cells in (1.0, 2.0, 3.0 if dim == 2 else np.sqrt(3.0)):
        _check(_cols(q * step + offset), _cols(grid * step + offset), cells * step)


@pytest.mark.parametrize("offset", [0.0, 1000.0])
@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("nq", [40, 5000])
def test_shell_of_near_misses(gpu, nq, dim, offset):
    rng = np.random.default_rng(nq + dim)
    radius = 0.125
    centre = rng.integers(0, 8, (40, dim)) / 4.0 + offset
    v = rng.normal(size=(12000, dim))
    v /= np.linalg.norm(v, axis=1, keepdims=True)
    off = 10.0 ** rng.uniform(-17, -3, 12000) * rng.choice([-1.0, 0.0, 1.0], 12000)
    p = centre[rng.integers(0, 40, 12000)] + v * (radius * (1.0 + off))[:, None]
    _check(_cols(centre[rng.integers(0, 40, nq)]), _cols(p), radius)
