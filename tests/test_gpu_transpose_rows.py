"""The device transpose on both sides of the line between a thread and a warp per
row (65,536 rows, 8 entries per row on average), with empty rows, duplicate
entries and weights: G^T P against float64."""
import numpy as np
import pytest
import scipy.sparse as sp

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_rows", [65535, 65536, 65700])
@pytest.mark.parametrize("per", [1, 7, 8])
def test_transposed_product(mm, n_rows, per):
    rng = np.random.default_rng(n_rows + per)
    n_cols, p = 3001, 5
    cnt = rng.integers(0, 2 * per + 1, n_rows)
    cnt[-1] += n_rows * per - cnt.sum() if cnt.sum() < n_rows * per else 0
    rp = np.concatenate([[0], np.cumsum(cnt)])
    ci = rng.integers(0, n_cols, rp[-1]).astype(np.int32)
    ci[1::5] = ci[:-1:5][:len(ci[1::5])]  # neighbours repeated: duplicates inside rows
    val = rng.uniform(0.5, 2.0, rp[-1]).astype(np.float32)
    P = rng.standard_normal((n_rows, p)).astype(np.float32)
    G = sp.csr_matrix((val.astype(np.float64), ci, rp), shape=(n_rows, n_cols))
    want = G.T @ P.astype(np.float64)
    got = mm.spmm(mm.CsrBlock(n_rows, n_cols, rp, ci, val), P, transpose=True)
    assert np.abs(got - want).max() < 1e-5 * np.abs(want).max()
