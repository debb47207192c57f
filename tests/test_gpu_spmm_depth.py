"""SpMM on both sides of the line between the 16-deep and the 4-deep gather
(155,648 threads: 19,456 rows at 8 lanes per row, 155,648 at one), with rows of 0
.. 69 nonzeros on both: the deep loop, the 4-wide one behind it and the tail."""
import numpy as np
import pytest
import scipy.sparse as sp

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,p", [(19455, 61), (19457, 61), (155647, 4), (155649, 4)])
def test_spmm_gather_depth_rows(mm, n, p):
    rng = np.random.default_rng(n)
    cnt = np.arange(n) % 70
    rp = np.concatenate([[0], np.cumsum(cnt)])
    G = sp.csr_matrix((np.ones(rp[-1]), rng.integers(0, 500, rp[-1]), rp), shape=(n, 500))
    P = rng.standard_normal((500, p)).astype(np.float32)
    G.sum_duplicates()
    want = G @ P.astype(np.float64)
    got = mm.spmm(mm.CsrBlock.from_scipy(G), P)
    assert np.abs(got - want).max() < 1e-5 * np.abs(want).max()
