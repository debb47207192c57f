"""The eigensolver at the sizes where its kernels change form: columns per lane
of the one-CTA Jacobi (16, 32, 56, 72 columns; more than 48 KB of shared memory
from 87).  Device against numpy in FP64.

Tolerances: those of the smaller sizes (test_gpu_whiten_sizes.py)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def rel(a, b):
    return np.abs(np.asarray(a) - np.asarray(b)).max() / max(np.abs(np.asarray(b)).max(), 1e-300)


def check(mm, n):
    rng = np.random.default_rng(n)
    B = rng.standard_normal((n, n))
    A = B @ B.T + 0.1 * np.eye(n)
    ev, V = mm.symeig(A)
    assert np.abs(V.T @ V - np.eye(n)).max() < 1e-10
    assert rel(ev, np.linalg.eigvalsh(A)[::-1]) < 1e-9
    assert np.abs(A @ V - V * ev).max() / np.abs(A).max() < 1e-9
    assert np.all(np.diff(ev) <= 0)


@pytest.mark.parametrize("n", [16, 56, 57, 72, 73, 86, 87, 95])
def test_symeig_one_cta(mm, n):
    check(mm, n)
