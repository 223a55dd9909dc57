"""Brute-force kNN over rows that are stored in an order, so that more rows of one range come near a query than the
first block of its record list holds: further blocks from the pool, and queries scanned again in short stages where the
pool has none left.  nbpg_test_gt_redone is nbpg_gt with a limit on those blocks and the number of such queries."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
ALL = 0xFFFFFFFF


def _gt(lib, base, q, dtype, metric, k, exact, blocks):
    from nbpg_gb300 import _lib
    from nbpg_gb300.index import _p
    ids, ds, redone = np.empty((len(q), k), np.uint32), np.empty((len(q), k), np.float32), C.c_uint32()
    _lib.check(lib.nbpg_test_gt_redone(_lib.DTYPES[dtype], _lib.METRICS[metric], base.shape[1], base.ctypes.data,
                                       len(base), q.ctypes.data, len(q), k, int(exact), _p(ids), _p(ds, _lib._f32p), 0,
                                       blocks, C.byref(redone)))
    return ids, ds, redone.value


def _redone(lib, base, q, dtype, metric, k, exact, limits):
    """How many queries were scanned again with each limit on the blocks; all results as DP4A gives them"""
    from nbpg_gb300.index import ground_truth
    want = ground_truth(base, q, dtype, metric, k=k, exact=exact, engine="dp4a")
    out = []
    for blocks in limits:
        ids, ds, redone = _gt(lib, base, q, dtype, metric, k, exact, blocks)
        assert np.array_equal(ids, want[0]) and np.array_equal(ds.view(np.uint32), want[1].view(np.uint32)), (metric, blocks)
        out.append(redone)
    return out


@pytest.mark.parametrize("exact", [False, True])
@pytest.mark.parametrize("dtype,dims,k", [("u8", 32, 10), ("u8", 300, 100), ("i8", 96, 128), ("u4", 40, 48)])
def test_gt_rows_stored_by_cluster(gpu_lib, dtype, dims, k, exact):
    """Both widths of a query tile, lists of many blocks, a pool that runs out at once and on the way, the two rules;
    the same rows in random order take one pass."""
    r = np.random.default_rng(dims)
    n, nq, centres = 120000, 2300, 4
    lab = r.integers(0, centres, n + nq)
    c = r.integers(40, 216, (centres, dims))
    x = np.clip(c[lab] + r.normal(scale=12.0, size=(n + nq, dims)), 0, 255).astype(np.uint8)
    if dtype == "i8":
        x = (x.astype(np.int16) - 128).astype(np.int8)
    q, rows = np.ascontiguousarray(x[n:]), x[:n]
    ordered = np.ascontiguousarray(rows[np.argsort(lab[:n], kind="stable")])
    for metric in ("l2", "ip"):
        every, some, none = _redone(gpu_lib, ordered, q, dtype, metric, k, exact, (ALL, 300, 0))
        assert every <= some <= none and (none > 0 or metric == "ip")
    assert _redone(gpu_lib, np.ascontiguousarray(rows), q, dtype, "l2", k, exact, (ALL,)) == [0]


@pytest.mark.parametrize("nq,step", [(2300, 5), (16700, 3), (16700, 1), (300, 299), (1, 1)])
def test_gt_some_queries_again(gpu_lib, nq, step):
    """Rows that come closer and closer to every step-th query (of one batch and of two, the last query among them),
    which are scanned again, and farther from the others."""
    r = np.random.default_rng(nq)
    b = r.integers(0, 256, (150000, 16)).astype(np.uint8)
    b = np.ascontiguousarray(b[np.argsort(-(b.astype(np.int32) ** 2).sum(1), kind="stable")])
    q = np.full((nq, 16), 255, np.uint8)
    near = np.arange(nq - 1, -1, -step)
    q[near] = r.integers(0, 3, (len(near), 16))
    for exact in (False, True):
        redone = _redone(gpu_lib, b, q, "u8", "l2", 10, exact, (ALL, 0))
        assert redone[1] == len(near), redone


@pytest.mark.parametrize("n,dims,nq,k", [(1171, 256, 1, 100), (1172, 256, 1, 100), (390, 256, 2, 16), (391, 256, 2, 16),
                                         (390, 256, 2, 17), (129, 130, 1, 128), (300, 576, 40, 10)])
def test_gt_small_calls_with_and_without_a_workspace(gpu_lib, n, dims, nq, k):
    """The sizes around which a call without a workspace goes to DP4A instead of allocating one"""
    import torch
    from nbpg_gb300.index import ground_truth_device, gt_workspace_size
    stride = (dims + 15) // 16 * 16
    g = torch.Generator(device="cuda").manual_seed(n)
    x = torch.randint(0, 256, (n + nq, stride), generator=g, device="cuda", dtype=torch.uint8)
    x[:, dims:] = 0
    ws = torch.empty(gt_workspace_size("u8", dims, n, nq, k), dtype=torch.uint8, device="cuda")
    assert ws.numel() > 0
    torch.cuda.synchronize()
    for exact in (False, True):
        out = []
        for w, engine in ((ws, "auto"), (None, "auto"), (None, "dp4a")):
            ids = torch.empty((nq, k), dtype=torch.int32, device="cuda")
            ds = torch.empty((nq, k), dtype=torch.float32, device="cuda")
            ground_truth_device(x.data_ptr(), n, x[n:].data_ptr(), nq, dims, stride, "u8", "l2", k, ids.data_ptr(),
                                ds.data_ptr(), exact=exact, engine=engine, d_workspace=w.data_ptr() if w is not None else 0,
                                workspace_bytes=ws.numel() if w is not None else 0)
            out.append((ids, ds))
        for ids, ds in out[1:]:
            assert torch.equal(ids, out[0][0]) and torch.equal(ds, out[0][1]), exact
