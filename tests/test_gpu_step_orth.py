"""The step's QR where the pivots of its Cholesky do not show how close to
dependent the columns are: a unit upper triangular matrix with -c above the
diagonal has pivot ratios above 1 / (1 + c^2 k), but a condition number of about
(1 + c)^k.  With a step width of 1e-30 the step returns the Q factor of Phi0.

Tolerances: Q^T Q = I to 1e-5 as in the other tests of the step; Cholesky QR with
a second pass is backward stable, so Q^T Phi0 is upper triangular to FP32
round-off of k terms, 6e-8 k, times 10, of Phi0's norm."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [33, 64, 100, 128, 160, 208])
@pytest.mark.parametrize("cond", [1e2, 1e3, 1e4, 1e5])
def test_hidden_condition(mm, oracle, k, cond):
    rng = np.random.default_rng(k)
    c = cond ** (1.0 / (k - 1)) - 1.0
    x = oracle.qr_pos(rng.standard_normal((k, k))) @ (np.eye(k) - c * np.triu(np.ones((k, k)), 1))
    x = x.astype(np.float32).astype(np.float64)
    nx = 64
    y = {n: rng.standard_normal((k, nx)) for n in ("Da", "Db", "Dc")}
    y.update({n + "_mu": y[n].mean(axis=1) for n in ("Da", "Db", "Dc")})
    e = mm.CsrBlock(nx, 1, np.zeros(nx + 1, np.int64), np.zeros(0, np.int32))
    o = mm.CsrBlock(1, 1, np.zeros(2, np.int64), np.zeros(0, np.int32))
    with mm.Pipeline(k=k, alpha0=1.0, stpm_method=mm.STPM_ONLINE, sweeps=1, minibatch=nx,
                     lr0=1e-30) as p:
        p.upload(mm.Graph([e, e, e, o, o], (nx, 1, 1, 1))).set_whitened(y).stpm(x)
        phi = p.phi()
    assert np.abs(phi.T @ phi - np.eye(k)).max() < 1e-5
    # (the tensor value's sign may have turned columns)
    assert np.abs(np.tril(phi.T @ x, -1)).max() < 6e-7 * k * np.linalg.norm(x, 2)


def test_step_flops(mm):
    """What is counted is what runs: 3 k^3 per step, 10/3 k^3 per exact pass and
    4 k^3 once for the first step's Phi (Phi^T Phi)^.2."""
    k, nx = 40, 400
    rng = np.random.default_rng(1)
    y = {n: rng.standard_normal((k, nx)) for n in ("Da", "Db", "Dc")}
    y.update({n + "_mu": y[n].mean(axis=1) for n in ("Da", "Db", "Dc")})
    e = mm.CsrBlock(nx, 1, np.zeros(nx + 1, np.int64), np.zeros(0, np.int32))
    o = mm.CsrBlock(1, 1, np.zeros(2, np.int64), np.zeros(0, np.int32))
    with mm.Pipeline(k=k, alpha0=1.0, stpm_method=mm.STPM_ONLINE, sweeps=2, minibatch=100) as p:
        p.upload(mm.Graph([e, e, e, o, o], (nx, 1, 1, 1))).set_whitened(y).stpm()
        s = p.stats()
    assert s["stpm_steps"] == 8
    assert s["step_flops"] == pytest.approx(k ** 3 * (3 * 8 + 10 / 3 * s["orth_passes"] + 4))
