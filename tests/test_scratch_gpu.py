"""Device memory and shared-memory limits as the library asks the CUDA runtime for them: child processes with
tests/runtime_shim.c between the two."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))
HEAD = """
import ctypes as C, sys
import numpy as np
sys.path[:0] = [{root!r}, {here!r}]
shim = C.CDLL(None)
shim.shim_limit.argtypes = [C.c_size_t]
shim.shim_used.restype = shim.shim_peak.restype = C.c_size_t
from nbpg_gb300 import _lib, synth
from nbpg_gb300.index import Index, LaunchConfig, QueryParams, ground_truth
r = np.random.default_rng(3)
""".format(root=os.path.dirname(HERE), here=HERE)


@pytest.fixture(scope="session")
def shim(gpu_lib, tmp_path_factory):
    so = tmp_path_factory.mktemp("shim") / "shim.so"
    subprocess.run(["gcc", "-O1", "-shared", "-fPIC", "-o", str(so), os.path.join(HERE, "runtime_shim.c"), "-ldl",
                    "-lpthread"], check=True)

    def run(code):
        p = subprocess.run([sys.executable, "-c", HEAD + code], env=dict(os.environ, LD_PRELOAD=str(so)),
                           capture_output=True, text=True, timeout=300)
        assert p.returncode == 0, p.stdout[-2000:] + p.stderr[-3000:]
    return run


def test_rerank_of_one_short_query_stays_in_its_scratch(shim):
    shim("""
base = r.integers(0, 256, (500, 16)).astype(np.uint8)
raw = r.normal(size=(500, 5)).astype(np.float32)
idx = Index(base, "u8", "l2", max_degree=16)
idx.build_vamana(L=24, VL=32, num_split=0, num_passes=1)
idx.set_raw_points(raw)
qp = QueryParams(k=1, beamSize=16)
many = idx.search_rerank(base[:64], raw[:64], qp, 1)
for i in range(3):
    one = idx.search_rerank(base[i:i + 1], raw[i:i + 1], qp, 1)
    assert one.ids[0, 0] == many.ids[i, 0] and one.dists[0, 0] == many.dists[i, 0]
idx.close()
assert shim.shim_peak() > 0 and shim.shim_overrun() == 0
""")


def test_shared_memory_limits_are_never_lowered(shim):
    """A kernel's limit belongs to every call of the process: one that needs less leaves it alone."""
    shim("""
def build(n, dims, R, L, VL, metric, fgim=False):
    idx = Index(r.integers(0, 256, (n, dims)).astype(np.uint8), "u8", metric, max_degree=R)
    (idx.build_fgim if fgim else idx.build_vamana)(L=L, VL=VL, num_split=2 if fgim else 0, num_passes=2 if fgim else 1)
    idx.close()
for dims, R, L, VL in [(256, 48, 90, 140), (64, 16, 24, 32), (256, 48, 90, 140)]:
    for metric in ("l2", "ip"):
        build(600, dims, R, L, VL, metric)
    build(600, dims, R, L, VL, "l2", fgim=True)
for dims, k in [(400, 100), (128, 100), (16, 1), (700, 150), (700, 3)]:
    rows = r.integers(0, 256, (900, dims)).astype(np.uint8)
    for engine in ("auto", "dp4a") + (("tensor",) if dims <= 128 else ()):
        ground_truth(rows, rows[:40], "u8", "l2", k=k, engine=engine)
for L in (90, 24):
    idx = Index(r.integers(0, 256, (600, 64)).astype(np.uint8), "u8", "l2", max_degree=16)
    h, _ = idx.build_hnsw(L=L, VL=190)
    h.close()
    idx.close()
assert shim.shim_peak() > 0 and shim.shim_lowered() == 0
""")


def test_knn_runs_in_the_memory_it_has(shim):
    """One query over 200k rows within the rows' own copies and 64 MB; with no room for any list, AUTO runs on DP4A
    and the explicit tensor engine says so."""
    shim("""
base = r.integers(0, 256, (200000, 128)).astype(np.uint8)
want = ground_truth(base, base[:1], "u8", "l2", k=100, engine="dp4a")
shim.shim_limit(base.nbytes * 3 + (64 << 20))
got = ground_truth(base, base[:1], "u8", "l2", k=100, engine="tensor")
assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1])
shim.shim_limit(base.nbytes + (1 << 20))
got = ground_truth(base, base[:1], "u8", "l2", k=100)
assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1])
try:
    ground_truth(base, base[:1], "u8", "l2", k=100, engine="tensor")
    raise SystemExit("no refusal")
except _lib.NbpgError as e:
    assert e.status == 2
shim.shim_limit(1 << 40)
got = ground_truth(base, base[:1], "u8", "l2", k=100)
assert np.array_equal(got[0], want[0]) and shim.shim_overrun() == 0 and shim.shim_peak() > 0
""")


@pytest.mark.parametrize("fgim", [False, True])
def test_build_leaves_out_what_does_not_fit(shim, fgim):
    """The neighbours' distances (n x R x 4 bytes) and the insert's key buffers only make the build faster: with less
    memory than they take the build runs without them and gives the same graph, until what it needs does not fit."""
    shim(f"fgim = {fgim}" + """
n, R = 20000, 32
base, _ = synth.u8_mixture(n, 1, dim=32, n_centres=32)
def build(limit):
    idx = Index(base, "u8", "l2", max_degree=R)
    shim.shim_limit(limit)
    shim.shim_reset_peak()
    try:
        (idx.build_fgim if fgim else idx.build_vamana)(L=40, VL=60, num_split=2 if fgim else 0, num_passes=2)
        g = idx.get_graph()
        return shim.shim_peak(), [tuple(r[1:1 + r[0]]) for r in g]
    except _lib.NbpgError as e:
        assert e.status == 2
        return None
    finally:
        shim.shim_limit(1 << 40)
        idx.close()
peak, want = build(1 << 40)
room = n * R * 4
for limit in (peak - 1, peak - room // 2, peak - room):
    used, got = build(limit)
    assert used <= limit and got == want
assert build(peak // 3) is None
assert build(1 << 40)[1] == want and shim.shim_overrun() == 0
""")


def test_get_graph_leaves_the_destination_to_the_copy(shim):
    """A destination that the host cannot write is answered by the copy's status, and the process lives on."""
    shim("""
g = np.zeros((300, 9), np.uint32)
g[:, 0], g[:, 1:4] = 3, r.integers(0, 300, (300, 3))
idx = Index(r.integers(0, 256, (300, 16)).astype(np.uint8), "u8", "l2", max_degree=8, graph=g)
other = Index(r.integers(0, 256, (4000, 16)).astype(np.uint8), "u8", "l2", max_degree=8)
device = other.device_info()[2]
status = _lib.lib().nbpg_index_get_graph(idx._h, C.cast(C.c_void_p(device), C.POINTER(C.c_uint32)), 0, 300)
assert status in (0, 3), status
live = np.arange(8)[None, :] < g[:, :1]
got = idx.get_graph()
assert np.array_equal(got[:, 0], g[:, 0]) and np.array_equal(got[:, 1:][live], g[:, 1:][live])
idx.close()
other.close()
""")


@pytest.mark.parametrize("kernel", ["batched", "plain"])
def test_search_runs_with_the_scratch_there_is(shim, kernel):
    """Long beams keep a visited filter per warp in global memory: with less of it the grids are smaller and the results
    the same."""
    shim(f"kernel = {kernel!r}" + """
base, q = synth.u8_mixture(4000, 600, dim=32, n_centres=24)
idx = Index(base, "u8", "ip", max_degree=24)
idx.build_vamana(L=32, VL=48, num_split=0, num_passes=1)
for L in (300, 200):
    qp = QueryParams(k=50, beamSize=L)
    idx2 = Index(base, "u8", "ip", max_degree=24, graph=idx.get_graph())
    want = idx2.search(q, qp, launch=LaunchConfig(kernel=kernel))
    idx2.close()
    for room in (100 << 20, 20 << 20, 4 << 20):  # (one CTA of 16 warps takes 2.6 MB at L = 300)
        idx2 = Index(base, "u8", "ip", max_degree=24, graph=idx.get_graph())
        shim.shim_limit(shim.shim_used() + room)
        for _ in range(2):
            got = idx2.search(q, qp, launch=LaunchConfig(kernel=kernel))
            for a, b in zip((want.ids, want.dists, want.count, want.visited, want.cmps),
                            (got.ids, got.dists, got.count, got.visited, got.cmps)):
                assert np.array_equal(a, b), (L, room)
        shim.shim_limit(1 << 40)
        idx2.close()
idx.close()
assert shim.shim_overrun() == 0
""")


@pytest.mark.parametrize("kernel", ["batched", "plain"])
def test_beam_above_the_calls_is_refused_for_all_its_queries(gpu_lib, kernel):
    """Inner product, a call of L = 19: the visited list of its exact re-run holds 160 entries, 8 per beam place.  A query
    that asks for L = 21 is answered with an empty row whether or not it would have been run again."""
    import numpy as np
    import torch
    from conftest import dataset
    from nbpg_gb300.index import Index, LaunchConfig, QueryParams
    base, q, g = dataset("i8", "ip")
    idx = Index(base, "i8", "ip", max_degree=g.shape[1] - 1, graph=g)
    rs, nq, k = idx.device_info()[1], len(q), 10
    d = torch.zeros((nq, rs), dtype=torch.uint8, device="cuda")
    d[:, :q.shape[1]] = torch.from_numpy(np.ascontiguousarray(q).view(np.uint8)).cuda()
    Ls = torch.tensor([19, 20, 21] * nq, dtype=torch.int32, device="cuda")[:nq].contiguous()
    ids = torch.full((nq, k), 7, dtype=torch.int32, device="cuda")
    counts = torch.full((3, nq), 7, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    idx.search_device(d.data_ptr(), nq, QueryParams(k=k, beamSize=19), ids.data_ptr(), k, None, counts[0].data_ptr(),
                      counts[1].data_ptr(), counts[2].data_ptr(), launch=LaunchConfig(kernel=kernel), d_Ls=Ls.data_ptr())
    torch.cuda.synchronize()
    refused = (Ls == 21).cpu().numpy()
    got, found = ids.cpu().numpy(), counts[0].cpu().numpy()
    assert (got[refused] == -1).all() and (found[refused] == 0).all()
    assert (found[~refused] > 0).all() and (got[~refused, 0] >= 0).all()
