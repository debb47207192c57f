"""Whitening at the sizes where its kernels change form: k (and the 2 k columns
of the sketches) at and beside the block sizes of the orthogonalisation, the
triangular factors and the eigensolver (8, 16, 32, 48, 64), and the sparse
products on both sides of the number of rows from which a row's gather is 4
instead of 16 deep.  Device against the FP64 oracle.

Tolerances: those of the golden comparisons (W and the factors of the
pseudo-inverses 1e-4 after the best rotation, products 1e-5 of the output's
scale); eigenpairs 1e-9, orthogonality 1e-10."""
import numpy as np
import pytest
import scipy.sparse as sp

from conftest import procrustes_align

pytestmark = pytest.mark.gpu


def rel(a, b):
    return np.abs(np.asarray(a) - np.asarray(b)).max() / max(np.abs(np.asarray(b)).max(), 1e-300)


@pytest.mark.parametrize("k", [1, 4, 8, 9, 16, 17, 24, 25, 31, 33, 48, 49])
def test_whitening_sizes(mm, oracle, k):
    rng = np.random.default_rng(k)
    n = 40 * k + 61
    z = [rng.integers(0, k, n) for _ in range(4)]

    def block(a, b):
        return sp.csr_matrix((rng.random((n, n)) < np.where(a[:, None] == b[None, :], 0.6, 0.02))
                             .astype(np.float64))

    Gxa, Gxb, Gxc = (block(z[0], z[q]) for q in (1, 2, 3))
    Gba, Gca = block(z[2], z[1]), block(z[3], z[1])
    g = mm.Graph([mm.CsrBlock.from_scipy(m) for m in (Gxa, Gxb, Gxc, Gba, Gca)], (n, n, n, n))
    sketches = [rng.standard_normal((n, 2 * k)).astype(np.float32).astype(np.float64)
                for _ in range(3)]
    with mm.Pipeline(k=k, alpha0=1.0) as p:
        p.upload(g).whiten(sketches)
        wh = p.whitening()
    ref = oracle.second_whiten(Gxa, Gxb, Gxc, k, 1.0, sketches)
    assert rel(procrustes_align(ref["W"], wh["W"]), ref["W"]) < 1e-4
    for a, b in (("Zb1", "Zb2"), ("Zc1", "Zc2")):
        assert rel(wh[a] @ wh[b], ref[a] @ ref[b]) < 1e-4


@pytest.mark.parametrize("n", [1, 2, 15, 17, 32, 33, 63, 65, 96, 97, 129])
def test_symeig_sizes(mm, n):
    rng = np.random.default_rng(n)
    B = rng.standard_normal((n, n))
    A = B @ B.T + 0.1 * np.eye(n)
    ev, V = mm.symeig(A)
    assert np.abs(V.T @ V - np.eye(n)).max() < 1e-10
    assert rel(ev, np.linalg.eigvalsh(A)[::-1]) < 1e-9
    assert np.abs(A @ V - V * ev).max() / np.abs(A).max() < 1e-9
    assert np.all(np.diff(ev) <= 0)


# rows of 0 .. 69 nonzeros; 155,648 threads is the line between the two forms
@pytest.mark.parametrize("n,p", [(70, 3), (155647, 4), (155649, 4), (9727, 61), (9729, 61)])
def test_spmm_gather_depth(mm, n, p):
    rng = np.random.default_rng(n)
    cnt = np.arange(n) % 70 if n < 20000 else np.arange(n) % 5
    rp = np.concatenate([[0], np.cumsum(cnt)])
    G = sp.csr_matrix((np.ones(rp[-1]), rng.integers(0, 500, rp[-1]), rp), shape=(n, 500))
    P = rng.standard_normal((500, p)).astype(np.float32)
    G.sum_duplicates()
    assert rel(mm.spmm(mm.CsrBlock.from_scipy(G), P), G @ P.astype(np.float64)) < 1e-5
