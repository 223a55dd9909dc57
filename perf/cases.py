"""What this framework is timed on: searches, graph builds, brute-force kNN and PCA encoding, each
through the entry point that a program calls, from one query to the 10k x 1M kNN.

Rows are seeded mixtures of the shapes and value ranges of `nbpg_gb300.synth`, made on the GPU.
Ids are returned as int32 (the bits of the unsigned ids), since torch indexes those everywhere.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from nbpg_gb300 import _lib
from nbpg_gb300.index import (Index, LaunchConfig, QueryParams, ground_truth_device, gt_workspace_size)

NIBBLES = ("u4", "i4")


def listed():
    return [
        # one query against a 100k index: the latency of a single lookup
        {"name": "search_one", "kind": "search", "n": 100_000, "dims": 128, "dtype": "u8", "metric": "l2", "R": 64,
         "nq": 1, "L": 32, "k": 10, "kernel": "plain", "lane_width": 4, "uneven": False},
        # the headline workload: 10k queries against 1M x 128 u8 at the beam that reaches recall 0.95
        {"name": "search_10k_1m", "kind": "search", "n": 1_000_000, "dims": 128, "dtype": "u8", "metric": "l2",
         "R": 64, "nq": 10_000, "L": 19, "k": 10, "kernel": "plain", "lane_width": 4, "uneven": False},
        # recommendation-style retrieval: inner product, requests that differ in beam and k, persistent kernel
        {"name": "search_uneven_ip", "kind": "search", "n": 250_000, "dims": 96, "dtype": "i8", "metric": "ip",
         "R": 64, "nq": 20_000, "L": 256, "k": 100, "kernel": "batched", "lane_width": 0, "uneven": True},
        # 4-bit PCA codes at a high-recall beam, the default launch
        {"name": "search_4bit", "kind": "search", "n": 250_000, "dims": 32, "dtype": "u4", "metric": "l2", "R": 48,
         "nq": 10_000, "L": 80, "k": 10, "kernel": "batched", "lane_width": 0, "uneven": False},
        # quantised search, then exact distances of the raw float rows, host arrays in and out
        {"name": "rerank_host", "kind": "rerank", "n": 100_000, "dims": 128, "R": 64, "nq": 2_000, "L": 50, "k": 10,
         "factor": 3},
        # a small collection with an odd row length, built from host rows
        {"name": "build_small_ip", "kind": "build", "n": 20_011, "dims": 100, "dtype": "i8", "metric": "ip", "R": 32,
         "L": 64, "VL": 96, "passes": 1, "split": 0, "dynamic": False},
        # a one-pass Vamana index of 100k rows
        {"name": "build_vamana_100k", "kind": "build", "n": 100_000, "dims": 128, "dtype": "u8", "metric": "l2",
         "R": 64, "L": 100, "VL": 140, "passes": 1, "split": 0, "dynamic": False},
        # the full NBPG recipe: split stage, popularity pass, dynamic prune, repair
        {"name": "build_nbpg_250k", "kind": "build", "n": 250_000, "dims": 128, "dtype": "u8", "metric": "l2",
         "R": 64, "L": 100, "VL": 140, "passes": 2, "split": 4, "dynamic": True},
        # ground truth of the headline workload, CompGT's admission rule
        {"name": "knn_10k_1m", "kind": "knn", "n": 1_000_000, "nq": 10_000, "dims": 128, "dtype": "u8",
         "metric": "l2", "k": 100, "exact": False},
        # ground truth of a small signed inner-product set, exact top k, odd sizes
        {"name": "knn_small_ip", "kind": "knn", "n": 50_003, "nq": 1_000, "dims": 96, "dtype": "i8", "metric": "ip",
         "k": 10, "exact": True},
        # long rows
        {"name": "knn_wide", "kind": "knn", "n": 200_000, "nq": 2_000, "dims": 256, "dtype": "u8", "metric": "l2",
         "k": 100, "exact": True},
        # float rows to packed 4-bit PCA-64 codes
        {"name": "pca_1m_4bit", "kind": "pca", "n": 1_000_000, "d_in": 128, "d_out": 64, "in_dtype": "f32",
         "out_dtype": "u4"},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["search", "search", "search", "rerank", "build", "build", "knn", "knn", "knn", "pca"])
    if kind == "search":
        dtype = rng.choice(["u8", "u8", "i8", "u4", "i4"])
        uneven = rng.random() < 0.3
        L = 256 if uneven else _log(rng, 10, 250)
        kernel = "batched" if uneven or L > 160 else rng.choice(["batched", "plain"])
        return {"kind": kind, "n": _log(rng, 20_000, 300_000),
                "dims": rng.randint(24, 64) if dtype in NIBBLES else rng.randint(48, 160), "dtype": dtype,
                "metric": rng.choice(["l2", "l2", "ip"]), "R": rng.choice([32, 48, 64]), "nq": _log(rng, 1, 10_000),
                "L": L, "k": 100 if uneven else min(L, rng.choice([1, 10, 10, 100])), "kernel": kernel,
                "lane_width": rng.choice([0, 4]), "uneven": uneven}
    if kind == "rerank":
        return {"kind": kind, "n": _log(rng, 20_000, 150_000), "dims": rng.randint(48, 160), "R": rng.choice([32, 64]),
                "nq": _log(rng, 1, 5_000), "L": _log(rng, 20, 150), "k": 10, "factor": rng.choice([0, 2, 3])}
    if kind == "build":
        passes = rng.choice([1, 2])
        dtype = rng.choice(["u8", "u8", "i8", "u4"])
        return {"kind": kind, "n": _log(rng, 1_000, 100_000),
                "dims": rng.randint(24, 64) if dtype in NIBBLES else rng.randint(48, 160), "dtype": dtype,
                "metric": rng.choice(["l2", "l2", "ip"]), "R": rng.choice([24, 32, 48, 64]), "L": rng.randint(32, 110),
                "VL": rng.randint(80, 160), "passes": passes, "split": rng.choice([0, 4]) if passes == 2 else 0,
                "dynamic": passes == 2 and rng.random() < 0.7}
    if kind == "knn":
        dtype = rng.choice(["u8", "u8", "i8", "u4", "i4"])
        nib = dtype in NIBBLES
        wide = rng.random() < 0.35
        dims = rng.randint(65, 200) if nib and wide else rng.randint(16, 64) if nib else \
            rng.randint(129, 400) if wide else rng.randint(32, 128)
        return {"kind": kind, "n": _log(rng, 5_000, 150_000 if wide else 600_000),
                "nq": _log(rng, 1, 2_000 if wide else 8_000), "dims": dims, "dtype": dtype,
                "metric": rng.choice(["l2", "l2", "ip"]), "k": rng.choice([1, 10, 50, 100]),
                "exact": rng.random() < 0.5}
    return {"kind": "pca", "n": _log(rng, 1_000, 1_000_000), "d_in": rng.randint(32, 192),
            "d_out": 2 * rng.randint(12, 32), "in_dtype": rng.choice(["f32", "f32", "u8", "i8"]),
            "out_dtype": rng.choice(["f32", "u8", "i8", "u4", "i4"])}


# ---------------------------------------------------------------------------
# inputs, from the seed alone
# ---------------------------------------------------------------------------
def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed) & 0x7FFFFFFFFFFF)


def _mixture(g, sizes, dims, lo, hi, sigma, centres=1000):
    """Float rows of a Gaussian mixture: one tensor per size, all around the same centres."""
    c = torch.rand(centres, dims, generator=g, device="cuda") * (hi - lo) + lo
    out = []
    for n in sizes:
        x = torch.randn(n, dims, generator=g, device="cuda") * sigma
        x += c[torch.randint(centres, (n,), generator=g, device="cuda")]
        out.append(x)
    return out


def _quantised(g, sizes, dims, dtype):
    """Rows as the library takes them: `dims` bytes each (4-bit codes two to a byte)."""
    if dtype == "u8":
        return [x.round_().clamp_(0, 255).to(torch.uint8) for x in _mixture(g, sizes, dims, 0.0, 120.0, 20.0)]
    if dtype == "i8":  # unit vectors scaled to 127
        xs = _mixture(g, sizes, dims, -1.0, 1.0, 0.35)
        return [(x / x.norm(dim=1, keepdim=True) * 127.0).round_().clamp_(-127, 127).to(torch.int8) for x in xs]
    xs = [x.round_().clamp_(0, 15).to(torch.uint8) for x in _mixture(g, sizes, 2 * dims, 2.0, 13.0, 1.5)]
    return [((x[:, 0::2] << 4) | x[:, 1::2]).contiguous() for x in xs]


def _padded(x, stride):
    if x.shape[1] == stride:
        return x.contiguous()
    y = torch.zeros(x.shape[0], stride, dtype=x.dtype, device=x.device)
    y[:, :x.shape[1]] = x
    return y


def _stride(dims):
    return (dims + 15) // 16 * 16


_STREAM = []


def _stream():
    """The one stream that the device-buffer calls of this program use."""
    if not _STREAM:
        _STREAM.append(torch.cuda.Stream())
    return _STREAM[0].cuda_stream


def _searchable(rows, dtype, metric, R):
    """An index over the rows with a graph as a serving program would load it."""
    idx = Index(rows.cpu().numpy(), dtype, metric, max_degree=R)
    idx.build_vamana(L=64, VL=96, num_split=0, num_passes=1, max_alpha=1.2)
    return idx


def prepare(case, seed):
    g = _generator(seed)
    s = {"case": case}
    kind = case["kind"]
    if kind == "search":
        rows, q = _quantised(g, [case["n"], case["nq"]], case["dims"], case["dtype"])
        nq, k = case["nq"], case["k"]
        s["index"] = _searchable(rows, case["dtype"], case["metric"], case["R"])
        s["queries"] = _padded(q, s["index"].device_info()[1])
        s["params"] = QueryParams(k=k, beamSize=case["L"])
        s["launch"] = LaunchConfig(kernel=case["kernel"], lane_width=case["lane_width"])
        s["Ls"] = s["ks"] = None
        if case["uneven"]:
            pick = torch.randint(4, (nq,), generator=g, device="cuda")
            s["Ls"] = torch.tensor([32, 64, 128, 256], dtype=torch.int32, device="cuda")[pick]
            ks = torch.tensor([1, 10, 100], dtype=torch.int32, device="cuda")
            s["ks"] = torch.minimum(ks[torch.randint(3, (nq,), generator=g, device="cuda")], s["Ls"])
        s["ids"] = torch.empty(nq, k, dtype=torch.int32, device="cuda")
        s["dists"] = torch.empty(nq, k, dtype=torch.float32, device="cuda")
        s["counts"] = torch.empty(3, nq, dtype=torch.int32, device="cuda")
        s["stream"] = _stream()
    elif kind == "rerank":
        raw, q = _mixture(g, [case["n"], case["nq"]], case["dims"], 0.0, 120.0, 20.0)
        s["index"] = _searchable(raw.round().clamp_(0, 255).to(torch.uint8), "u8", "l2", case["R"])
        s["index"].set_raw_points(raw.cpu().numpy())
        s["raw"] = q.cpu().numpy()
        s["queries"] = q.round().clamp_(0, 255).to(torch.uint8).cpu().numpy()
        s["params"] = QueryParams(k=case["k"], beamSize=case["L"])
    elif kind == "build":
        s["rows"] = _quantised(g, [case["n"]], case["dims"], case["dtype"])[0].cpu().numpy()
    elif kind == "knn":
        rows, q = _quantised(g, [case["n"], case["nq"]], case["dims"], case["dtype"])
        s["base"], s["queries"] = (_padded(x, _stride(case["dims"])) for x in (rows, q))
        need = gt_workspace_size(case["dtype"], case["dims"], case["n"], case["nq"], case["k"])
        s["workspace"] = torch.empty(max(need, 16), dtype=torch.uint8, device="cuda")
        s["ids"] = torch.empty(case["nq"], case["k"], dtype=torch.int32, device="cuda")
        s["dists"] = torch.empty(case["nq"], case["k"], dtype=torch.float32, device="cuda")
        s["stream"] = _stream()
    else:
        s["rows"], s["mat"], s["bias"] = _pca_inputs(g, case)
        wide = case["d_out"] // 2 if case["out_dtype"] in NIBBLES else case["d_out"]
        s["codes"] = torch.empty(case["n"], wide, device="cuda",
                                 dtype=torch.float32 if case["out_dtype"] == "f32" else torch.uint8)
        s["stream"] = _stream()
    return s


def _pca_inputs(g, case):
    d_in, d_out = case["d_in"], case["d_out"]
    if case["in_dtype"] == "f32":
        rows = _mixture(g, [case["n"]], d_in, -3.5, 3.5, 1.0)[0]
    else:
        rows = _quantised(g, [case["n"]], d_in, case["in_dtype"])[0]
    # an orthogonal projection scaled so that three standard deviations of the rows map to 1
    x = rows[:4096].float()
    basis = torch.linalg.qr(torch.randn(d_in, d_in, generator=g, device="cuda"))[0]
    basis = basis[torch.arange(d_out, device="cuda") % d_in]
    mat = (basis / (3.0 * (x @ basis.T).std(dim=0) + 1e-3)[:, None]).contiguous()
    return rows.contiguous(), mat, -(mat @ x.mean(dim=0))


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "search":
        c = s["counts"]
        s["index"].search_device(s["queries"].data_ptr(), case["nq"], s["params"], s["ids"].data_ptr(), case["k"],
                                 s["dists"].data_ptr(), c[0].data_ptr(), c[1].data_ptr(), c[2].data_ptr(),
                                 stream=s["stream"], launch=s["launch"],
                                 d_Ls=None if s["Ls"] is None else s["Ls"].data_ptr(),
                                 d_ks=None if s["ks"] is None else s["ks"].data_ptr())
        return {"ids": s["ids"], "dists": s["dists"], "counts": c}
    if kind == "rerank":
        r = s["index"].search_rerank(s["queries"], s["raw"], s["params"], case["factor"])
        return {"ids": r.ids.view(np.int32), "dists": r.dists,
                "counts": [x.view(np.int32) for x in (r.count, r.visited, r.cmps)]}
    if kind == "build":
        idx = Index(s["rows"], case["dtype"], case["metric"], max_degree=case["R"])
        st, _, _ = idx.build_vamana(L=case["L"], VL=case["VL"], num_split=case["split"], num_passes=case["passes"],
                                    min_alpha=1.05 if case["dynamic"] else 1.0,
                                    max_alpha=1.1 if case["dynamic"] else 1.2, dynamic_prune=case["dynamic"])
        graph = idx.get_graph()
        idx.close()
        return {"graph": graph.view(np.int32), "isolated": int(st.isolated)}
    if kind == "knn":
        ground_truth_device(s["base"].data_ptr(), case["n"], s["queries"].data_ptr(), case["nq"], case["dims"],
                            s["base"].shape[1], case["dtype"], case["metric"], case["k"], s["ids"].data_ptr(),
                            s["dists"].data_ptr(), exact=case["exact"], d_workspace=s["workspace"].data_ptr(),
                            workspace_bytes=s["workspace"].numel(), stream=s["stream"])
        return {"ids": s["ids"], "dists": s["dists"]}
    lib = _lib.lib()
    _lib.check(lib.nbpg_pca_encode_device(_lib.DTYPES[case["in_dtype"]], s["rows"].data_ptr(), case["n"],
                                          case["d_in"], s["mat"].data_ptr(), s["bias"].data_ptr(), case["d_out"],
                                          _lib.DTYPES[case["out_dtype"]], s["codes"].data_ptr(), s["stream"]))
    return s["codes"]


def _search_work(nq, L, R, dims, n):
    """A beam search expands about L + 10 nodes; each gives its adjacency row (half full) and leaves
    about 500 + 10 L rows in all to compare (both measured on 1M x 128 mixtures)."""
    expanded, compared = min(n, L + 10), min(n, 500 + 10 * L)
    return {"bytes": nq * (expanded * (2 * R + 4) + (compared + 1) * dims), "flops": nq * compared * 2 * dims}


def work(case):
    kind = case["kind"]
    if kind in ("search", "rerank"):
        L = 120 if case.get("uneven") else case["L"]  # the mean of 32, 64, 128 and 256
        w = _search_work(case["nq"], L, case["R"], case["dims"], case["n"])
        w["bytes"] += case["nq"] * (8 * case["k"] + 12)
        if kind == "rerank":
            w["bytes"] += case["nq"] * 4 * case["dims"] * min(L, case["k"] * max(1, case["factor"]))
        return w
    if kind == "build":
        # per insert: a search, about 24 pair distances per kept edge, the row written twice
        inserts = case["n"] * (case["passes"] + (2 if case["split"] else 0))
        w = _search_work(inserts, case["L"], case["R"], case["dims"], case["n"])
        w["bytes"] += inserts * (24 * case["R"] * case["dims"] + 8 * case["R"])
        w["flops"] += inserts * 24 * case["R"] * 2 * case["dims"]
        return w
    if kind == "knn":
        n, nq, dims = case["n"], case["nq"], case["dims"]
        return {"bytes": (n + nq) * dims + nq * case["k"] * 8,
                "flops": 2 * n * nq * dims * (2 if case["dtype"] in NIBBLES else 1)}
    n, d_in, d_out = case["n"], case["d_in"], case["d_out"]
    out = {"f32": 4.0, "u4": 0.5, "i4": 0.5}.get(case["out_dtype"], 1.0)
    return {"bytes": n * (d_in * (4 if case["in_dtype"] == "f32" else 1) + out * d_out) + 4 * d_in * d_out,
            "flops": 2 * n * d_in * d_out}


def _elements(x, dtype):
    """Rows as float64 values; a 4-bit code counts 16 times its nibble, which is how distances read it."""
    if dtype in NIBBLES:
        x = torch.stack([x >> 4, x & 15], dim=2).reshape(x.shape[0], -1)
        return x.double() * 16.0
    return x.double()


def exact(case, seed):
    """Distances of the exact kNN and PCA values in 64 bits.  A beam search's, a build's and CompGT's
    results are which ids were met on the way, which no plain computation gives."""
    kind = case["kind"]
    g = _generator(seed)
    if kind == "knn" and case["exact"]:
        rows, q = (_elements(x, case["dtype"]) for x in
                   _quantised(g, [case["n"], case["nq"]], case["dims"], case["dtype"]))
        norms = (rows * rows).sum(1)
        out = []
        for b in range(0, q.shape[0], 256):
            d = -(q[b:b + 256] @ rows.T)
            if case["metric"] == "l2":
                d = norms[None, :] + 2.0 * d + (q[b:b + 256] ** 2).sum(1, keepdim=True)
            out.append(torch.topk(d, case["k"], dim=1, largest=False, sorted=True).values)
        return {"ids": None, "dists": torch.cat(out)}
    if kind == "pca" and case["out_dtype"] == "f32":
        rows, mat, bias = _pca_inputs(g, case)
        return rows.double() @ mat.double().T + bias.double()
    return None
