"""Timed workloads of the neighbor path, through the public entry points.

A case is a dict of plain values; ``listed()`` names the fixed ones and
``draw(rng)`` gives more of the same ranges.  ``prepare`` makes the inputs and
whatever a program holds before the call (resident scenes, prepared query
sets, captured graphs, output buffers), ``run`` makes one call as a program
does, ``work`` counts the bytes and operations the answer cannot do without
and ``exact`` recomputes the floating outputs in 64 bits with torch alone.

Kinds of case:

* ``host``     one drop-in kernel call: records in host memory, rows back in
               host memory (``prepare_b200(kernel).bind(...).run_raw()``);
* ``plain``    the same call on device records: scene build and rows;
* ``scene``    rows from a scene, resident or built in the call
               (``B200Scene.query_device``: fixed radius, bounded KNN, KNN);
* ``multi``    several fixed-radius requests against one resident scene;
* ``nearest``  directed Hausdorff: scene build, nearest distances, witness;
* ``batch``    many uneven problems: one build and one query for all;
* ``graph``    the captured graph over prepared problem batches;
* ``summary``  ranked summaries of a prepared query set on a resident scene;
* ``count``    fixed-radius counts, device columns in and out.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import rtdl_b200 as rt
from rtdl_b200.batch import B200ProblemBatch, B200ProblemBatchGraph
from rtdl_b200.runtime import (FRN_ROW_DTYPE, KNN_ROW_DTYPE, POINT2D_DTYPE, POINT3D_DTYPE, PackedPoints,
                               fixed_radius_neighbors_device)
from rtdl_b200.workloads import CLUSTERED_RADIUS


def listed():
    return [
        # the smallest call: 4,096 x 4,096 float64 points in 2D through the
        # kernel API, every point in radius kept; launches and latency count
        {"name": "host_frn_2d_4k", "kind": "host", "dim": 2, "dist": "uniform", "f64": True, "nq": 4096, "ns": 4096,
         "mean": 5.147, "pred": "fixed_radius_neighbors", "limit": 4096, "shuffle": False},
        # an ordinary kernel call: KNN of ragged clustered 3D sets, rows to the host
        {"name": "host_knn8_3d_60k", "kind": "host", "dim": 3, "dist": "clustered", "f64": False, "nq": 60013,
         "ns": 71993, "mean": 0.0, "pred": "knn_rows", "limit": 8, "shuffle": False},
        # the headline: 1M x 1M clustered 3D, radius for a mean of about 32
        # neighbors, at most 64 kept, scene build included
        {"name": "plain_frn_3d_1m", "kind": "plain", "dim": 3, "dist": "clustered", "f64": False, "nq": 1 << 20,
         "ns": 1 << 20, "mean": 32.0, "limit": 64, "shuffle": False},
        # KNN k = 16 on the same sets, scene build included
        {"name": "build_knn16_3d_1m", "kind": "scene", "resident": False, "dim": 3, "dist": "clustered", "f64": False,
         "nq": 1 << 20, "ns": 1 << 20, "mean": 0.0, "pred": "knn_rows", "limit": 16, "shuffle": False},
        # directed Hausdorff of two 4M-point 2D sets, scene build included
        {"name": "hausdorff_2d_4m", "kind": "nearest", "dim": 2, "nq": 1 << 22, "ns": 1 << 22},
        # uneven independent problems of 1,024 to 262,144 points, built and
        # answered together (the largest case: about 6M points a side)
        {"name": "batch_frn_128", "kind": "batch", "problems": 128, "lo": 1024, "hi": 262144},
        # the same kind of problems prepared once, answered by graph replays
        {"name": "graph_frn_64", "kind": "graph", "problems": 64, "lo": 1024, "hi": 262144},
        # a small served request (log-uniform sizes start at 100 probes)
        {"name": "served_frn_3d_311", "kind": "scene", "resident": True, "dim": 3, "dist": "clustered", "f64": False,
         "nq": 311, "ns": 2000003, "mean": 32.0, "pred": "fixed_radius_neighbors", "limit": 64, "shuffle": False},
        # several served requests of uneven sizes in one launch sequence
        {"name": "served_frn_multi_6", "kind": "multi", "dim": 3, "dist": "clustered", "f64": False, "requests": 6,
         "lo": 100, "hi": 400000, "ns": 800011, "mean": 24.0, "limit": 64},
        # a served KNN request with the longest list the traces ask for
        {"name": "served_knn32_3d_100k", "kind": "scene", "resident": True, "dim": 3, "dist": "clustered",
         "f64": False, "nq": 100003, "ns": 1000003, "mean": 0.0, "pred": "knn_rows", "limit": 32, "shuffle": False},
        # the published ranked-summary benchmark's densest set: 262,144 points
        # in 8 Gaussian clusters, r = 0.02, k_max = 50 (hundreds in radius)
        {"name": "summary_3d_262k", "kind": "summary", "dist": "rtnn", "n": 262144, "radius": 0.02, "limit": 50},
        # density counts over 2D device columns with a threshold (outlier and
        # DBSCAN-style core flags)
        {"name": "count_2d_1m", "kind": "count", "nq": 1000003, "ns": 1 << 20, "mean": 24.0, "threshold": 16},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["host", "plain", "scene", "scene", "scene", "multi", "nearest", "batch", "graph", "summary",
                       "count"])
    if kind in ("host", "plain"):
        top = 40_000 if kind == "host" else 1 << 20
        dim = rng.choice([2, 3])
        c = {"kind": kind, "dim": dim, "dist": rng.choice(["uniform", "clustered"]), "f64": rng.random() < 0.4,
             "nq": _log(rng, 1000, top), "ns": _log(rng, 1000, top), "mean": rng.uniform(2.0, 48.0)}
        if kind == "host":
            c["pred"] = rng.choice(["fixed_radius_neighbors", "fixed_radius_neighbors", "bounded_knn_rows", "knn_rows"])
        c["limit"] = rng.choice([1, 8, 16, 32]) if c.get("pred") == "knn_rows" else rng.choice([16, 33, 64])
        c["shuffle"] = rng.random() < 0.3
        return c
    if kind == "scene":
        pred = rng.choice(["fixed_radius_neighbors", "bounded_knn_rows", "knn_rows", "knn_rows"])
        return {"kind": kind, "resident": rng.random() < 0.7, "dim": rng.choice([2, 3, 3]),
                "dist": rng.choice(["uniform", "clustered"]), "f64": rng.random() < 0.25, "nq": _log(rng, 100, 1 << 20),
                "ns": _log(rng, 100_000, 1 << 21), "mean": rng.uniform(8.0, 48.0), "pred": pred,
                "limit": rng.choice([1, 4, 8, 16, 32] if pred == "knn_rows" else [16, 50, 64]),
                "shuffle": rng.random() < 0.2}
    if kind == "multi":
        return {"kind": kind, "dim": rng.choice([2, 3, 3]), "dist": rng.choice(["uniform", "clustered"]),
                "f64": rng.random() < 0.2, "requests": rng.randint(2, 12), "lo": 100, "hi": _log(rng, 1000, 400_000),
                "ns": _log(rng, 100_000, 1 << 21), "mean": rng.uniform(8.0, 40.0), "limit": rng.choice([16, 64])}
    if kind == "nearest":
        return {"kind": kind, "dim": rng.choice([2, 3]), "nq": _log(rng, 10_000, 1 << 22),
                "ns": _log(rng, 10_000, 1 << 22)}
    if kind in ("batch", "graph"):
        return {"kind": kind, "problems": _log(rng, 4, 128 if kind == "batch" else 64), "lo": 1024,
                "hi": rng.choice([16384, 65536, 262144])}
    if kind == "summary":
        return {"kind": kind, "dist": rng.choice(["uniform", "shell", "rtnn"]), "n": _log(rng, 20_000, 262_144),
                "radius": 0.02, "limit": rng.choice([16, 50, 64])}
    return {"kind": kind, "nq": _log(rng, 2000, 1 << 20), "ns": _log(rng, 2000, 1 << 21),
            "mean": rng.uniform(4.0, 64.0), "threshold": rng.choice([0, 5, 16])}


# ---- inputs -----------------------------------------------------------------

def _gen(seed, stream):
    g = torch.Generator(device="cuda")
    g.manual_seed((seed * 1009 + stream) % (1 << 62))
    return g


def _rand(g, *shape):
    return torch.rand(*shape, generator=g, dtype=torch.float64, device="cuda")


def _randn(g, *shape):
    return torch.randn(*shape, generator=g, dtype=torch.float64, device="cuda")


def _points(dist, n, dim, f64, seed, stream):
    """(n, dim) float64 on the GPU; FP32-exact values unless f64."""
    g = _gen(seed, stream)
    if dist == "uniform":
        p = _rand(g, n, dim)
    elif dist == "clustered":  # 64 Gaussian clusters and a 10% uniform background
        centres = _rand(_gen(seed, 0), 64, dim)
        which = torch.randint(0, 64, (n,), generator=g, device="cuda")
        p = centres[which] + 0.01 * _randn(g, n, dim)
        bg = _rand(g, n) < 0.1
        p = torch.where(bg[:, None], _rand(g, n, dim), p).clamp_(0.0, 1.0)
    elif dist == "rtnn":  # 8 clusters, sigma 0.035
        centres = 0.12 + 0.76 * _rand(_gen(seed, 0), 8, dim)
        which = torch.arange(n, device="cuda") % 8
        p = (centres[which] + 0.035 * _randn(g, n, dim)).clamp_(0.0, 1.0)
    else:  # a thin spherical shell
        v = _randn(g, n, 3)
        r = (0.34 + 0.025 * _randn(g, n, 1)).clamp_(0.0, 0.49)
        p = 0.5 + r * v / v.norm(dim=1, keepdim=True)
    return p if f64 else p.float().double()


def _radius(c, ns, mean):
    dim = c["dim"]
    if c["dist"] == "clustered":
        if dim == 3:
            return CLUSTERED_RADIUS * ((1 << 20) / ns * mean / 32.0) ** (1.0 / 3.0)
        # 64 clusters of sigma 0.01: a cluster point's mean density in 2D
        return math.sqrt(mean / (ns * 0.9 / 64.0) * 4.0 * 0.01 ** 2)
    return math.sqrt(mean / (ns * math.pi)) if dim == 2 else (mean / (ns * 4.0 / 3.0 * math.pi)) ** (1.0 / 3.0)


def _ids(n, shuffle, seed, stream):
    if shuffle:
        return torch.randperm(n, generator=_gen(seed, stream), device="cuda")
    return torch.arange(n, device="cuda")


def _records(points, ids):
    """Device records in the ABI layout: (n, dim + 1) float64 with the id in the first slot's low half."""
    return torch.cat([ids.to(torch.int64).view(torch.float64)[:, None], points], dim=1).contiguous()


def _packed(records):
    dim = records.shape[1] - 1
    host = records.cpu().numpy().reshape(-1).view(POINT3D_DTYPE if dim == 3 else POINT2D_DTYPE)
    return PackedPoints(records=host, count=len(host), dimension=dim)


def _ranked(c):
    return c["pred"] != "fixed_radius_neighbors"


def _host_capacity(c):
    """Rows the program makes room for: every query's limit, or four times the expected number and some."""
    return int(c["nq"] * min(c["limit"], 64.0 + 4.0 * c["mean"]))


def _sets(c, seed):
    """(query points, query ids, search points, search ids)."""
    q = _points(c["dist"], c["nq"], c["dim"], c["f64"], seed, 1)
    s = _points(c["dist"], c["ns"], c["dim"], c["f64"], seed, 2)
    return q, _ids(c["nq"], c.get("shuffle"), seed, 3), s, _ids(c["ns"], c.get("shuffle"), seed, 4)


def _nearest_sets(c, seed):
    """A uniform set and its jittered copy (or a jittered sample of it) with 1% of the points displaced."""
    ns, nq, dim = c["ns"], c["nq"], c["dim"]
    b = _points("uniform", ns, dim, False, seed, 1)
    g = _gen(seed, 2)
    a = b[torch.arange(nq, device="cuda") % ns] + 1e-3 * _randn(g, nq, dim)
    moved = _rand(g, nq) < 0.01
    a = torch.where(moved[:, None], _rand(g, nq, dim), a).float().double()
    return a, b


def _problems(c, seed):
    """Problem sizes, offsets, points, radii: uniform points in boxes of random aspect ratio."""
    rng = np.random.default_rng(seed)
    m = c["problems"]
    span = (math.log(c["lo"]), math.log(c["hi"]))
    # sizes spread evenly over the logarithm, paired at random, so that every
    # seed has the same amount of work
    grid = np.exp(span[0] + (np.arange(m) + 0.5) / m * (span[1] - span[0])).astype(np.int64)
    nb, nq = grid[rng.permutation(m)], grid[rng.permutation(m)]
    scale = np.exp(rng.uniform(-1.0, 1.0, (m, 3)))
    mean = rng.uniform(8.0, 64.0, m)
    radius = (mean * scale.prod(axis=1) / (nb * 4.0 / 3.0 * math.pi)) ** (1.0 / 3.0)

    def side(counts, stream):
        counts_t = torch.from_numpy(counts).cuda()
        which = torch.repeat_interleave(torch.arange(m, device="cuda"), counts_t)
        pts = (_rand(_gen(seed, stream), int(counts.sum()), 3) * torch.from_numpy(scale).cuda()[which]).float().double()
        off = np.concatenate([[0], np.cumsum(counts)]).astype(np.uint64)
        start = torch.from_numpy(off[:-1].astype(np.int64)).cuda()[which]
        return pts, torch.arange(len(pts), device="cuda") - start, off

    s, sid, soff = side(nb, 2)
    q, qid, qoff = side(nq, 1)
    return q, qid, qoff, s, sid, soff, radius


def _requests(c, seed):
    """Query offsets of the requests: sizes spread evenly over the logarithm, in random order."""
    rng = np.random.default_rng(seed)
    m = c["requests"]
    span = (math.log(c["lo"]), math.log(c["hi"]))
    sizes = np.exp(span[0] + (np.arange(m) + 0.5) / m * (span[1] - span[0])).astype(np.int64)[rng.permutation(m)]
    return np.concatenate([[0], np.cumsum(sizes)]).astype(np.uint64)


def _kernel(c, radius):
    kind = rt.Points3D if c["dim"] == 3 else rt.Points
    pred, limit = c["pred"], c["limit"]
    fields = ["query_id", "neighbor_id", "distance"] + ([] if pred == "fixed_radius_neighbors" else ["neighbor_rank"])

    @rt.kernel(backend="rtdl", precision="float_approx")
    def neighbors():
        q = rt.input("query_points", kind, role="probe")
        s = rt.input("search_points", kind, role="build")
        if pred == "knn_rows":
            predicate = rt.knn_rows(k=limit)
        elif pred == "bounded_knn_rows":
            predicate = rt.bounded_knn_rows(radius=radius, k_max=limit)
        else:
            predicate = rt.fixed_radius_neighbors(radius=radius, k_max=limit)
        return rt.emit(rt.refine(rt.traverse(q, s, accel="bvh"), predicate=predicate), fields=fields)

    return rt.prepare_b200(neighbors)


class _Rows:
    """A device row buffer (16-B rows, or 24-B rows with ranks) and its columns."""

    def __init__(self, capacity, ranked):
        self.capacity, self.ranked = capacity, ranked
        words = 6 if ranked else 4
        self.buf = torch.zeros(capacity * words, dtype=torch.int32, device="cuda")
        w = self.buf.view(-1, words)
        self.qid, self.nid = w[:, 0], w[:, 1]
        self.dist = self.buf.view(torch.float64).view(-1, words // 2)[:, 1]
        self.rank = w[:, 4] if ranked else None
        self.address = self.buf.data_ptr()

    def columns(self, n):
        """The whole buffer, zero past its n rows."""
        out = {"count": n, "query_id": self.qid, "neighbor_id": self.nid, "distance": self.dist}
        if self.ranked:
            out["rank"] = self.rank
        return out


def prepare(case, seed):
    c, kind = case, case["kind"]
    st = {"case": c}
    if kind == "host":
        q, qid, s, sid = _sets(c, seed)
        kernel = _kernel(c, _radius(c, c["ns"], c["mean"]))
        st.update(kernel=kernel, q=_packed(_records(q, qid)), s=_packed(_records(s, sid)), view=None)
        if c["pred"] != "knn_rows":
            st["rows"] = np.zeros(_host_capacity(c), dtype=KNN_ROW_DTYPE if _ranked(c) else FRN_ROW_DTYPE)
    elif kind == "plain":
        q, qid, s, sid = _sets(c, seed)
        st.update(q=_records(q, qid), s=_records(s, sid), radius=_radius(c, c["ns"], c["mean"]),
                  rows=_Rows(c["nq"] * min(c["limit"], c["ns"]), False))
    elif kind == "scene":
        q, qid, s, sid = _sets(c, seed)
        st.update(q=_records(q, qid), s=_records(s, sid), radius=_radius(c, c["ns"], c["mean"]) if c["mean"] else 0.0,
                  rows=_Rows(c["nq"] * min(c["limit"], c["ns"]), _ranked(c)))
        torch.cuda.synchronize()
        if c["resident"]:
            st["scene"] = rt.B200Scene(None, dimension=c["dim"], device_points=(st["s"].data_ptr(), c["ns"]))
    elif kind == "multi":
        off = _requests(c, seed)
        q, qid, s, sid = _sets(dict(c, nq=int(off[-1])), seed)
        st.update(q=_records(q, qid), s=_records(s, sid), off=off, rows=_Rows(int(off[-1]) * c["limit"], False),
                  radius=_radius(c, c["ns"], c["mean"]) * np.linspace(0.8, 1.1, c["requests"]))
        torch.cuda.synchronize()
        st["scene"] = rt.B200Scene(None, dimension=c["dim"], device_points=(st["s"].data_ptr(), c["ns"]))
    elif kind == "nearest":
        q, s = _nearest_sets(c, seed)
        st.update(q=_records(q, _ids(c["nq"], False, seed, 3)), s=_records(s, _ids(c["ns"], False, seed, 4)),
                  nd=torch.zeros(c["nq"], dtype=torch.float64, device="cuda"),
                  ni=torch.zeros(c["nq"], dtype=torch.int32, device="cuda"))
    elif kind in ("batch", "graph"):
        q, qid, qoff, s, sid, soff, radius = _problems(c, seed)
        st.update(q=_records(q, qid), qoff=qoff, s=_records(s, sid), soff=soff, radius=radius,
                  rows=_Rows(len(q) * 64, False))
        torch.cuda.synchronize()
        if kind == "graph":
            st["batch"] = B200ProblemBatch(device_points=(st["s"].data_ptr(), soff), dimension=3)
            st["graph"] = B200ProblemBatchGraph([st["batch"]], st["q"].data_ptr(), qoff, radius=radius, k_max=64,
                                                rows_address=st["rows"].address, rows_capacity=st["rows"].capacity)
    elif kind == "summary":
        n = c["n"]
        p = _points(c["dist"], n, 3, False, seed, 1)
        st.update(s=_records(p, torch.arange(n, device="cuda")))
        st["out"] = torch.zeros(n * 5, dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        st["scene"] = rt.B200Scene(None, dimension=3, device_points=(st["s"].data_ptr(), n))
        st["queries"] = rt.B200Queries(dimension=3, device_points=(st["s"].data_ptr(), n))
    else:
        q = _points("uniform", c["nq"], 2, False, seed, 1)
        s = _points("uniform", c["ns"], 2, False, seed, 2)

        def columns(p):
            return {"ids": torch.arange(len(p), device="cuda", dtype=torch.int32), "x": p[:, 0].contiguous(),
                    "y": p[:, 1].contiguous()}

        st.update(q=columns(q), s=columns(s), radius=math.sqrt(c["mean"] / (c["ns"] * math.pi)),
                  out={k: torch.zeros(c["nq"], dtype=torch.int32, device="cuda")
                       for k in ("query_ids", "neighbor_counts", "threshold_flags")})
        torch.cuda.synchronize()
        st["prepared"] = rt.prepare_b200_fixed_radius_count_threshold_2d_device_search_columns(
            st["s"], max_radius=st["radius"])
    torch.cuda.synchronize()
    return st


def run(st):
    c = st["case"]
    kind = c["kind"]
    if kind == "host":
        if c["pred"] == "knn_rows":  # the rows are used where the library put them
            if st["view"] is not None:
                st["view"].close()
            st["view"] = st["kernel"].bind(query_points=st["q"], search_points=st["s"]).run_raw()
            rows = st["view"].to_numpy(copy=False)
            return {"query_id": rows["query_id"], "neighbor_id": rows["neighbor_id"], "distance": rows["distance"],
                    "rank": rows["neighbor_rank"]}
        rows = st["rows"]  # the rows are copied into the program's own array
        with st["kernel"].bind(query_points=st["q"], search_points=st["s"]).run_raw() as view:
            n = len(view)
            rows[:n].view(np.uint8)[:] = view.to_numpy(copy=False).view(np.uint8)
        out = {"count": n, "query_id": rows["query_id"], "neighbor_id": rows["neighbor_id"],
               "distance": rows["distance"]}
        if _ranked(c):
            out["rank"] = rows["neighbor_rank"]
        return out
    if kind == "plain":
        rows = st["rows"]
        n = fixed_radius_neighbors_device(st["q"].data_ptr(), c["nq"], st["s"].data_ptr(), c["ns"],
                                          dimension=c["dim"], radius=st["radius"], k_max=c["limit"],
                                          rows_address=rows.address, rows_capacity=rows.capacity)
        return rows.columns(n)
    if kind == "scene":
        rows = st["rows"]
        scene = st.get("scene") or rt.B200Scene(None, dimension=c["dim"], device_points=(st["s"].data_ptr(), c["ns"]))
        n = scene.query_device(st["q"].data_ptr(), c["nq"], predicate=c["pred"], radius=st["radius"], limit=c["limit"],
                               rows_address=rows.address, rows_capacity=rows.capacity)
        if not c["resident"]:
            scene.close()
        return rows.columns(n)
    if kind == "multi":
        rows = st["rows"]
        off = st["scene"].fixed_radius_neighbors_multi_device(
            st["q"].data_ptr(), st["off"], radius=st["radius"], k_max=c["limit"], rows_address=rows.address,
            rows_capacity=rows.capacity)
        return {"row_offsets": off.astype(np.int64), **rows.columns(int(off[-1]))}
    if kind == "nearest":
        with rt.B200Scene(None, dimension=c["dim"], device_points=(st["s"].data_ptr(), c["ns"])) as scene:
            r = scene.directed_hausdorff_device(st["q"].data_ptr(), c["nq"], nearest_id_address=st["ni"].data_ptr(),
                                                nearest_distance_address=st["nd"].data_ptr())
        return {"nearest_distance": st["nd"], "nearest_id": st["ni"], "distance": r["distance"],
                "source_id": r["source_id"], "target_id": r["target_id"]}
    if kind == "batch":
        rows = st["rows"]
        with B200ProblemBatch(device_points=(st["s"].data_ptr(), st["soff"]), dimension=3) as batch:
            off = batch.fixed_radius_neighbors_device(st["q"].data_ptr(), st["qoff"], radius=st["radius"], k_max=64,
                                                      rows_address=rows.address, rows_capacity=rows.capacity)
        return {"row_offsets": off.astype(np.int64), **rows.columns(int(off[-1]))}
    if kind == "graph":
        off, status = st["graph"].replay()
        return {"row_offsets": off.astype(np.int64), "status": status, **st["rows"].columns(int(off[-1]))}
    if kind == "summary":
        agg = st["scene"].ranked_summaries_prepared(st["queries"], radius=c["radius"], k_max=c["limit"],
                                                    summaries_address=st["out"].data_ptr())
        words = st["out"].view(torch.int32).view(-1, 10)
        values = st["out"].view(-1, 5)
        return {"query_id": words[:, 0], "neighbor_count": words[:, 1], "nearest_id": words[:, 2],
                "kth_id": words[:, 3], "nearest_distance": values[:, 2], "kth_distance": values[:, 3],
                "sum_distance": values[:, 4], "aggregate": agg}
    out = st["out"]
    st["prepared"].write_device_count_threshold_columns(st["q"], radius=st["radius"], threshold=c["threshold"],
                                                        query_ids_out=out["query_ids"],
                                                        neighbor_counts_out=out["neighbor_counts"],
                                                        threshold_flags_out=out["threshold_flags"])
    return dict(out)


def work(case):
    c, kind = case, case["kind"]
    if kind in ("batch", "graph"):
        m, span = c["problems"], (math.log(c["lo"]), math.log(c["hi"]))
        n = sum(int(math.exp(span[0] + (i + 0.5) / m * (span[1] - span[0]))) for i in range(m))
        nq, ns, dim, found, row = n, n, 3, 34.0, 16
    elif kind == "multi":
        m, span = c["requests"], (math.log(c["lo"]), math.log(c["hi"]))
        nq = sum(int(math.exp(span[0] + (i + 0.5) / m * (span[1] - span[0]))) for i in range(m))
        ns, dim, found, row = c["ns"], c["dim"], c["mean"], 16
    elif kind == "summary":
        nq = ns = c["n"]
        dim, found, row = 3, 1.0, 40
    elif kind == "count":
        nq, ns, dim, found, row = c["nq"], c["ns"], 2, 1.0, 12
    elif kind == "nearest":
        nq, ns, dim, found, row = c["nq"], c["ns"], c["dim"], 1.0, 12
    else:
        pred = c.get("pred", "fixed_radius_neighbors")
        nq, ns, dim = c["nq"], c["ns"], c["dim"]
        found = min(c["limit"], ns) if pred == "knn_rows" else min(c["limit"], c["mean"])
        row = 16 if pred == "fixed_radius_neighbors" else 24
    record = (dim + 1) * 8
    return {"bytes": (nq + ns) * record + nq * found * row, "flops": nq * found * 3 * dim}


# ---- the floating outputs in 64 bits ------------------------------------------

_ROOM = 1 << 26  # pairs of one dense tile


def _d2(q, s):
    """Squared distances of every pair, axes added in order."""
    d = s[None, :, 0] - q[:, None, 0]
    acc = d * d
    for a in range(1, q.shape[1]):
        d = s[None, :, a] - q[:, None, a]
        acc += d * d
    return acc


def _windows(q, s, half):
    """Tiles of queries along x with the search points within `half` of them: (query index, search index)."""
    qx, qo = torch.sort(q[:, 0])
    sx, so = torch.sort(s[:, 0])
    at, step = 0, 1024
    while at < len(q):
        end = min(len(q), at + step)
        lo = int(torch.searchsorted(sx, qx[at] - half))
        hi = int(torch.searchsorted(sx, qx[end - 1] + half, right=True))
        if (end - at) * max(1, hi - lo) > _ROOM and end - at > 1:
            step = max(1, step // 2)
            continue
        yield qo[at:end], so[lo:hi]
        at = end
        if (hi - lo) * step * 2 < _ROOM:
            step *= 2


def _padded(dist, capacity):
    out = torch.zeros(capacity, dtype=torch.float64, device=dist.device)
    out[: len(dist)] = dist
    return out


def _in_radius(q, qkey, s, sid, radius, limit):
    """(query key, distance, sid) of the `limit` nearest in radius, by (query key, distance, sid)."""
    rows, dist, ids = [], [], []
    for qi, si in _windows(q, s, radius * (1 + 1e-12)):
        d = _d2(q[qi], s[si]).sqrt_()
        hit = (d <= radius).nonzero()
        rows.append(qkey[qi[hit[:, 0]]])
        ids.append(sid[si[hit[:, 1]]])
        dist.append(d[hit[:, 0], hit[:, 1]])
    rows, dist, ids = torch.cat(rows), torch.cat(dist), torch.cat(ids)
    o = torch.sort(ids).indices  # stable sorts, least significant key first
    o = o[torch.sort(dist[o], stable=True).indices]
    o = o[torch.sort(rows[o], stable=True).indices]
    rows, dist, ids = rows[o], dist[o], ids[o]
    first = torch.searchsorted(rows, rows, side="left")
    keep = torch.arange(len(rows), device=rows.device) - first < limit
    return rows[keep], dist[keep], ids[keep]


def _k_nearest(q, s, k):
    """(nq, k) ascending distances of the k nearest."""
    k = min(k, len(s))
    out = torch.empty(len(q), k, dtype=torch.float64, device=q.device)
    left = torch.arange(len(q), device=q.device)
    half = 2.0 * (max(k, 4) / len(s)) ** (1.0 / q.shape[1])
    while len(left):
        again = []
        for qi, si in _windows(q[left], s, half):
            if len(si) < k:
                again.append(left[qi])
                continue
            d = torch.topk(_d2(q[left[qi]], s[si]), k, dim=1, largest=False).values.sort(dim=1).values.sqrt_()
            out[left[qi]] = d
            again.append(left[qi][d[:, -1] >= half * (1 - 1e-9)])
        if half > 4.0:
            break
        left, half = torch.cat(again), half * 4.0
    return out


def exact(case, seed):
    c, kind = case, case["kind"]
    if kind in ("host", "plain", "scene"):
        q, qid, s, sid = _sets(c, seed)
        pred = c.get("pred", "fixed_radius_neighbors")
        if pred == "knn_rows":
            dist = _k_nearest(q, s, c["limit"])[torch.argsort(qid)].reshape(-1)
            if kind == "host":
                return {"query_id": None, "neighbor_id": None, "distance": dist, "rank": None}
        else:
            dist = _in_radius(q, qid, s, sid, _radius(c, c["ns"], c["mean"]), c["limit"])[1]
        capacity = _host_capacity(c) if kind == "host" else c["nq"] * min(c["limit"], c["ns"])
        out = {"count": None, "query_id": None, "neighbor_id": None, "distance": _padded(dist, capacity)}
        return dict(out, rank=None) if pred != "fixed_radius_neighbors" else out
    if kind == "multi":
        off = _requests(c, seed)
        q, qid, s, sid = _sets(dict(c, nq=int(off[-1])), seed)
        radii = _radius(c, c["ns"], c["mean"]) * np.linspace(0.8, 1.1, c["requests"])
        parts = [_in_radius(q[int(a):int(b)], qid[int(a):int(b)], s, sid, float(r), c["limit"])[1]
                 for a, b, r in zip(off[:-1], off[1:], radii)]
        return {"row_offsets": None, "count": None, "query_id": None, "neighbor_id": None,
                "distance": _padded(torch.cat(parts), int(off[-1]) * c["limit"])}
    if kind == "nearest":
        q, s = _nearest_sets(c, seed)
        d = _k_nearest(q, s, 1)[:, 0]
        return {"nearest_distance": d, "nearest_id": None, "distance": float(d.max()), "source_id": None,
                "target_id": None}
    if kind in ("batch", "graph"):
        q, qid, qoff, s, sid, soff, radius = _problems(c, seed)
        parts = []
        for p in range(c["problems"]):
            qa, qb, sa, sb = int(qoff[p]), int(qoff[p + 1]), int(soff[p]), int(soff[p + 1])
            parts.append(_in_radius(q[qa:qb], qid[qa:qb], s[sa:sb], sid[sa:sb], float(radius[p]), 64)[1])
        out = {"row_offsets": None, "count": None, "query_id": None, "neighbor_id": None,
               "distance": _padded(torch.cat(parts), len(q) * 64)}
        return dict(out, status=None) if kind == "graph" else out
    if kind == "summary":
        n = c["n"]
        p = _points(c["dist"], n, 3, False, seed, 1)
        ids = torch.arange(n, device="cuda")
        rows, dist, _ = _in_radius(p, ids, p, ids, c["radius"], c["limit"])
        count = torch.bincount(rows, minlength=n)
        end = torch.cumsum(count, 0)
        total = torch.zeros(n, dtype=torch.float64, device="cuda").index_add_(0, rows, dist)
        return {"query_id": None, "neighbor_count": None, "nearest_id": None, "kth_id": None,
                "nearest_distance": dist[end - count], "kth_distance": dist[end - 1], "sum_distance": total,
                "aggregate": {"query_count": None, "bounded_neighbor_count": None, "nearest_id_checksum": None,
                              "kth_id_checksum": None, "sum_distance": float(dist.sum())}}
    return None
