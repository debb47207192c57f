"""The k x k step kernel and the reduction behind the power iteration at the
sizes where their layouts change: k at and beside multiples of 8 (blocks of the
Cholesky factorisation) and of the padded sizes (32 .. 208: one CTA at 32,
KP / 8 CTAs to 128, KP / 16 above).  Whitened data of the model with unit
noise, started near its components; device against the FP64 oracle.

Tolerance: FP32 products and 3xTF32 contractions perturb a step by about 1e-6
relative to y's scale, so 5 x the oracle's own response to a 1e-6 relative
perturbation of y, and at least 2e-5 (k FP32 round-offs of the entries of
Phi); a power iteration's lambda is the cube of a norm: three times that."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

KS = [1, 7, 8, 9, 16, 17, 31, 32, 33, 48, 49, 64, 65, 80, 81, 97, 112, 113, 128, 129, 160, 161,
      200, 208]


def rel(a, b):
    return float(np.linalg.norm(np.asarray(a) - np.asarray(b)) / np.linalg.norm(b))


def data(oracle, k, nx, seed):
    rng = np.random.default_rng(seed)
    comp = oracle.qr_pos(rng.standard_normal((k, k)))
    h = rng.dirichlet(np.full(k, 1.0 / k), size=nx) if k > 1 else np.ones((nx, 1))
    base = np.sqrt(2.0 * k) * h @ comp.T
    y = {n: (base + rng.standard_normal((nx, k))).astype(np.float32).astype(np.float64).T
         for n in ("Da", "Db", "Dc")}
    y.update({n + "_mu": y[n].mean(axis=1) for n in ("Da", "Db", "Dc")})
    phi0 = oracle.qr_pos(comp + 0.3 / np.sqrt(k) * rng.standard_normal((k, k)))
    noisy = {n: v * (1 + 1e-6 * rng.standard_normal(v.shape)) if n in ("Da", "Db", "Dc") else v
             for n, v in y.items()}
    return y, noisy, phi0


def pipeline(mm, k, nx, y, **cfg):
    e = mm.CsrBlock(nx, 1, np.zeros(nx + 1, np.int64), np.zeros(0, np.int32))
    o = mm.CsrBlock(1, 1, np.zeros(2, np.int64), np.zeros(0, np.int32))
    p = mm.Pipeline(k=k, alpha0=1.0, **cfg)
    p.upload(mm.Graph([e, e, e, o, o], (nx, 1, 1, 1))).set_whitened(y)
    return p


@pytest.mark.parametrize("k", KS)
def test_online_steps(mm, oracle, k):
    nx = 12 * k + 77
    b = -(-nx // 2)
    y, noisy, phi0 = data(oracle, k, nx, k)
    with pipeline(mm, k, nx, y, stpm_method=mm.STPM_ONLINE, sweeps=4, minibatch=b) as p:
        p.stpm(phi0)
        lam, phi = p.lam(), p.phi()
    assert np.abs(phi.T @ phi - np.eye(k)).max() < 1e-5
    lam_o, phi_o, _ = oracle.stpm_online(y, 1.0, phi0, sweeps=4, minibatch=b)
    lam_n, phi_n, _ = oracle.stpm_online(noisy, 1.0, phi0, sweeps=4, minibatch=b)
    assert rel(phi, phi_o) < max(2e-5, 5 * rel(phi_n, phi_o))
    assert rel(lam, lam_o) < max(2e-5, 5 * rel(lam_n, lam_o))


@pytest.mark.parametrize("k", [1, 31, 32, 33, 100, 128, 129, 208])
def test_power_iterations(mm, oracle, k):
    nx = 8 * k + 600
    y, noisy, phi0 = data(oracle, k, nx, 1000 + k)
    cfg = dict(min_iter=6, max_iter=6, tol=0.0)
    with pipeline(mm, k, nx, y, stpm_method=mm.STPM_BATCH_POWER, **cfg) as p:
        p.stpm(phi0)
        lam, phi, trace = p.lam(), p.phi(), p.convergence()
    args = dict(min_iter=6, max_iter=6, tol=0.0)
    lam_o, phi_o, it, err = oracle.tensor_decomp_batch(y, 1.0, phi0, **args)
    lam_n, phi_n, _, _ = oracle.tensor_decomp_batch(noisy, 1.0, phi0, **args)
    assert len(trace) == it
    assert abs(trace[-1] - err) < 1e-4 * max(err, 1e-2) + 2e-5 * np.sqrt(k)
    assert rel(phi, phi_o) < max(2e-5, 5 * rel(phi_n, phi_o))
    assert rel(lam, lam_o) < max(6e-5, 5 * rel(lam_n, lam_o))


# the adjoint contraction's thread groups: 8 up to k = 32, 4 to 64, 2 to 80
@pytest.mark.parametrize("k,nx", [(1, 65), (32, 431), (33, 500), (48, 1025), (64, 801), (65, 1000),
                                  (80, 1300)])
def test_adjoint_steps(mm, oracle, k, nx):
    b = -(-nx // 2)
    y, noisy, phi0 = data(oracle, k, nx, 2000 + k)
    with pipeline(mm, k, nx, y, stpm_method=mm.STPM_ADJOINT, sweeps=4, minibatch=b) as p:
        p.stpm(phi0)
        lam, phi = p.lam(), p.phi()
    lam_o, phi_o, _ = oracle.stpm_online(y, 1.0, phi0, sweeps=4, minibatch=b, adjoint=True)
    lam_n, phi_n, _ = oracle.stpm_online(noisy, 1.0, phi0, sweeps=4, minibatch=b, adjoint=True)
    assert rel(phi, phi_o) < max(2e-5, 5 * rel(phi_n, phi_o))
    assert rel(lam, lam_o) < max(2e-5, 5 * rel(lam_n, lam_o))
