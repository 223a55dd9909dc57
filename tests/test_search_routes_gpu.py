"""The sizes at which a search goes from one kernel to another (a few inner-product queries, long rows on the plain kernel,
four words a lane): every side of each line against the oracle."""
import numpy as np
import pytest

from conftest import dataset

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("metric", ["l2", "ip"])
@pytest.mark.parametrize("dims,lane_width", [(96, 0), (128, 4), (384, 0), (512, 0), (513, 0)])
def test_search_on_both_sides_of_each_line(gpu_lib, oracle_lib, metric, dims, lane_width):
    from nbpg_gb300.index import Index, LaunchConfig, QueryParams
    base, q, g = dataset("u8", metric, n=1500, dims=dims, nq=13, R=16, L=24)
    idx = Index(base, "u8", metric, max_degree=g.shape[1] - 1, graph=g)
    for L, k in [(32, 10), (33, 10), (63, 20), (64, 5), (128, 10), (129, 10)]:
        o = oracle_lib.search("u8", metric, base, g, q, L=L, k=k)
        for kernel in ("plain", "batched"):
            for nq in (1, 4, 5, 12, 13):
                r = idx.search(q[:nq], QueryParams(k=k, beamSize=L), launch=LaunchConfig(kernel=kernel, lane_width=lane_width))
                assert np.array_equal(r.ids, o[0][:nq]) and np.array_equal(r.dists, o[1][:nq]), (L, kernel, nq)
                assert np.array_equal(r.visited, o[3][:nq]) and np.array_equal(r.cmps, o[4][:nq]), (L, kernel, nq)
    idx.close()
