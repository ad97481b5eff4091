"""The workloads that the engine's timings are taken on.

Every case goes through the Python binding (rt-rknn_gb300/rknn.py), as a
caller's program does, over the generators of rt-rknn_gb300/datagen.py.  Sizes
are those of the five benchmark workloads (1k/10k, 100k/1M and 1M/10M uniform,
200k/4M clustered with ties, 20k/2M street layout with k from 1 to 100), and
draw() spreads over the same ranges, odd sizes included.

A case's fields: kind (the entry point), layout, nf and nu (points), nq
(queries of a pass), k (the largest where `mixed` is set: then every query has
its own, log-uniform from 1), mode (fp32 or fp64 predicates) and filter.

The results are user ids, which are exact on the float32 coordinates, so there
are no computed numbers that a 64-bit evaluation would approach.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.abspath("rt-rknn_gb300"))
import datagen  # noqa: E402
import rknn  # noqa: E402


def _case(name, kind, layout, nf, nu, nq, k, mode, filter="auto", mixed=False):
    c = {"kind": kind, "layout": layout, "nf": nf, "nu": nu, "nq": nq, "k": k, "mode": mode,
         "filter": filter, "mixed": mixed}
    return {"name": name, **c} if name else c


def listed():
    return [
        # the smallest calls: a small data set answered query by query in the
        # drop-in form (double-precision predicates, the influence zone)
        _case("single_small_fp64", "query", "uniform", 1000, 10_000, 8, 5, "fp64", "inf"),
        # the drop-in form at scale, as the command line runs it
        _case("single_zone_fp64", "query", "uniform", 100_000, 1_000_000, 8, 10, "fp64", "inf"),
        # a caller that needs one answer at a time and takes the default filter
        _case("single_fp32", "query", "uniform", 100_000, 1_000_000, 8, 10, "fp32"),
        # the benchmark's batch, host arrays in and out
        _case("batch_fp32", "batch", "uniform", 100_000, 1_000_000, 1000, 10, "fp32"),
        # the same batch with double-precision predicates
        _case("batch_fp64", "batch", "uniform", 100_000, 1_000_000, 1000, 10, "fp64"),
        # a batch through the reference's pruning, an odd number of queries
        _case("zone_batch_fp32", "batch", "uniform", 100_000, 1_000_000, 999, 10, "fp32", "inf"),
        # a pipeline that keeps queries and results on the GPU
        _case("device_batch_fp32", "device", "uniform", 100_000, 1_000_000, 16_384, 10, "fp32"),
        # skewed data with exact ties and duplicates: thousands of candidates
        # a query, many of them near a bisector
        _case("clustered_fp32", "batch", "clustered", 200_000, 4_000_000, 2000, 10, "fp32"),
        # a road-network layout, many queries with k from 1 to 100: millions
        # of result ids
        _case("street_fp32", "batch", "street", 20_000, 2_000_000, 16_384, 100, "fp32", mixed=True),
        # the same in double precision: the largest pass
        _case("street_fp64", "batch", "street", 20_000, 2_000_000, 16_384, 100, "fp64", mixed=True),
        # a burst of requests to the server over an index larger than the L2
        _case("serve_burst_fp32", "serve", "uniform", 1_000_000, 10_000_000, 512, 64, "fp32", mixed=True),
        # a new data set: the index built and its first batch answered
        _case("build_and_batch", "build", "uniform", 1_000_000, 10_000_000, 1000, 10, "fp32"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    what = rng.choice(["query", "batch", "batch", "zone", "device", "clustered", "street", "serve", "build"])
    mode = rng.choice(["fp32", "fp64"])
    if what == "clustered":
        nf = _log(rng, 2000, 200_000)
        return _case(None, "batch", "clustered", nf, int(nf * rng.uniform(5, 20)), _log(rng, 50, 2000),
                     rng.randint(1, 25), mode)
    if what == "street":
        nf = _log(rng, 1000, 20_000)
        return _case(None, "batch", "street", nf, int(nf * rng.uniform(10, 100)), _log(rng, 100, 16_384),
                     rng.randint(8, 100), mode, mixed=True)
    nf = _log(rng, 1000, 500_000)
    nu = int(nf * rng.uniform(5, 20))
    if what == "query":
        return _case(None, "query", "uniform", nf, nu, rng.randint(1, 8), rng.randint(1, 25), mode,
                     rng.choice(["auto", "inf"]))
    if what == "zone":
        return _case(None, "batch", "uniform", nf, nu, _log(rng, 10, 2000), rng.randint(1, 25), mode, "inf")
    if what == "serve":
        return _case(None, "serve", "uniform", nf, nu, _log(rng, 32, 512), rng.randint(4, 64), mode, mixed=True)
    if what == "build":
        return _case(None, "build", "uniform", nf, nu, _log(rng, 10, 1000), rng.randint(1, 25), "fp32")
    mixed = rng.random() < 0.3
    return _case(None, "batch" if what == "batch" else "device", "uniform", nf, nu, _log(rng, 10, 16_384),
                 rng.randint(1, 25), mode, mixed=mixed)


def _mean_k(case):
    """The mean k of a pass: with `mixed`, of floor(exp(U(0, log(k + 1))))."""
    k = case["k"]
    return sum(j * math.log((j + 1) / j) for j in range(1, k + 1)) / math.log(k + 1) if case["mixed"] else k


def _room(case):
    """Ids that the caller's output buffer holds: the mean number of results
    and what a pass's queries may exceed it by."""
    nq = case["nq"]
    return int(nq * _mean_k(case) * case["nu"] / case["nf"] * (1.25 + 8 / math.sqrt(nq))) + 65_536


def prepare(case, seed):
    nf, nu, nq, k = case["nf"], case["nu"], case["nq"], case["k"]
    seed = int(seed) & 0x7fffffff
    if case["layout"] == "street":
        ds = datagen.street(nu=nu, nf=nf, seed=seed, nq=nq, kmax=k)
    elif case["layout"] == "clustered":
        ds = datagen.gaussmix(nf, nu, seed=seed, nq=min(nq, nf), k=k)
    else:
        ds = datagen.uniform(nf, nu, seed=seed, nq=min(nq, nf), k=k)
    rng = np.random.default_rng([seed, 7])
    qs = ds.queries
    if qs.size < nq:                    # more queries than facilities: some asked again
        qs = np.concatenate([qs, rng.integers(0, nf, nq - qs.size)])
    ks = np.full(nq, k, np.int32)
    if case["mixed"]:
        ks = np.floor(np.exp(rng.uniform(0.0, math.log(k + 1), nq))).clip(1, k).astype(np.int32)
    s = {"kind": case["kind"], "mode": case["mode"], "filter": case["filter"], "k": k,
         "q": np.ascontiguousarray(qs, dtype=np.int32), "ks": ks, "off": np.zeros(nq + 1, np.int64)}
    if case["kind"] == "build":
        s["ds"] = ds
        s["ids"] = np.full(_room(case), -1, np.int32)
        return s
    idx = s["index"] = rknn.Index.of(ds, filter=case["filter"])
    if case["kind"] == "query":
        # the room of one answer: uniform points' regions are near their mean
        s["ids"] = np.full((nq, min(nu, 32 * k * nu // nf + 1024)), -1, np.int32)
    elif case["kind"] == "serve":
        s["server"] = rknn.Server(idx)
        s["ids"] = np.full(_room(case), -1, np.int32)
    elif case["kind"] == "device":
        # a pipeline on a stream of its own, results kept in its own tensor
        s["stream"] = torch.cuda.Stream()
        idx.set_stream(s["stream"].cuda_stream)
        s["d_q"] = torch.from_numpy(s["q"]).cuda()
        s["d_k"] = torch.from_numpy(ks).cuda()
        s["d_ids"] = torch.full((_room(case),), -1, dtype=torch.int32, device="cuda")
        torch.cuda.synchronize()
    else:
        # a page-locked id buffer kept for every batch, passed once before
        # the work begins: from then on the kernels write into it
        s["ids"] = rknn.pinned_ids(_room(case))
        _batch(s, 1)
        s["ids"].fill(-1)
    return s


class _Device:
    """A view of the engine's device memory for torch; the tensor made from it
    keeps the index, which owns that memory, alive."""

    def __init__(self, idx, ptr, n):
        self.owner = idx
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": "<i4", "data": (ptr, False), "version": 3}


def _batch(s, nq):
    """rknn_query_batch (include/rknn_gpu.h) into the caller's buffers."""
    ids, off = s["ids"], s["off"]
    mode = rknn.MODE_FP64 if s["mode"] == "fp64" else rknn.MODE_FP32
    rc = rknn.load().rknn_query_batch(s["index"].h, s["q"].ctypes.data, s["ks"].ctypes.data, nq, mode,
                                      ids.ctypes.data, ids.size, off.ctypes.data, None)
    if rc != 0:
        raise RuntimeError(rknn.load().rknn_last_error().decode())
    return ids, off


def run(s):
    """Ids and offsets, in the caller's buffers: what lies past the last
    result is as prepare() left it."""
    kind, mode, off = s["kind"], s["mode"], s["off"]
    if kind == "batch":
        return _batch(s, s["q"].size)
    if kind == "query":
        idx, k, ids = s["index"], s["k"], s["ids"]
        for i, q in enumerate(s["q"]):
            got = idx.query(q, k, mode)
            off[i + 1] = off[i] + got.size
            ids[i, :got.size] = got
        return ids, off
    if kind == "device":
        idx, nq = s["index"], s["d_q"].numel()
        with torch.cuda.stream(s["stream"]):
            idx.query_batch_device(s["d_q"].data_ptr(), s["d_k"].data_ptr(), nq, s["k"], mode)
            p_ids, p_off = idx.device_results()
            d_off = torch.as_tensor(_Device(idx, p_off, nq + 1), device="cuda").clone()
            n = int(d_off[nq])
            if n:
                s["d_ids"][:n].copy_(torch.as_tensor(_Device(idx, p_ids, n), device="cuda"))
        return s["d_ids"], d_off
    if kind == "serve":
        srv, ids = s["server"], s["ids"]
        tickets = [srv.submit(q, k, mode) for q, k in zip(s["q"].tolist(), s["ks"].tolist())]
        at = 0
        for i, t in enumerate(tickets):
            got = srv.wait(t)
            ids[at:at + got.size] = got
            at += got.size
            off[i + 1] = at
        return ids, off
    with rknn.Index.of(s["ds"], filter=s["filter"]) as idx:
        got, o = idx.query_batch_flat(s["q"], s["ks"], mode)
        s["ids"][:got.size] = got
        off[:] = o
    return s["ids"], off


def work(case):
    """Every result id has to be written and its user's coordinates and id
    read once; each query reads its index and k and the facilities that bound
    its region (about 6k of them), and a user is accepted once the about k/2
    facilities nearer to it than q are told from the others: 5 operations a
    distance.  Every user lies in the sets of its k nearest facilities, so a
    query's set has k nu/nf members on average."""
    nf, nu, nq = case["nf"], case["nu"], case["nq"]
    k = _mean_k(case)
    results = nq * k * nu / nf
    b = 8 * nq + 12 * min(nu, results) + 8 * min(nf, 6 * k * nq) + 4 * results + 8 * (nq + 1)
    f = results * 5 * (k / 2 + 1)
    if case["kind"] == "build":         # points and ids in, the same out in cell order
        b += 24 * (nf + nu)
        f += 4 * (nf + nu)
    return {"bytes": b, "flops": f}
