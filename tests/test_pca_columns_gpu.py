"""PCA encode on both sides of the row count from which 34 to 48 outputs take a block of 48 columns."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,d_out", [(8191, 34), (8192, 34), (8192, 48), (65, 48), (8191, 50)])
@pytest.mark.parametrize("kout", ["f32", "u4"])
def test_encode_columns_by_rows(gpu_lib, oracle_lib, n, d_out, kout):
    from nbpg_gb300.pca import encode
    r = np.random.default_rng(n + d_out)
    x = r.normal(size=(n, 70)).astype(np.float32)
    mat = (r.normal(size=(d_out, 70)) * 0.1).astype(np.float32)
    bias = (r.normal(size=d_out) * 0.1).astype(np.float32)
    assert np.array_equal(encode(x, mat, bias, kout), oracle_lib.pca_encode(x, mat, bias, kout))
