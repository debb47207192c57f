"""X^T X with one panel, the form that the Cholesky QR runs: on the tensor cores
the 128 x 128 tiles below the diagonal are left out and read mirrored, and a
diagonal tile stages its operand once.  The products and their order are those
of the general form (two copies of the panel), so every entry is that form's, bit
for bit, the mirrored tiles' those of the tile above the diagonal.  One to three
tiles and their edges."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [4096, 5003])
@pytest.mark.parametrize("pa", [64, 80, 127, 128, 129, 200, 256, 257, 300])
def test_one_panel(mm, n, pa):
    rng = np.random.default_rng(n + pa)
    A = (rng.standard_normal((n, pa)) * np.linspace(0.2, 5.0, pa)).astype(np.float32)
    want = mm.gram(A, A.copy(), alpha=0.5)
    i, j = np.meshgrid(np.arange(pa) // 128, np.arange(pa) // 128, indexing="ij")
    want = np.where(i > j, want.T, want)
    assert np.array_equal(mm.gram(A, A, alpha=0.5), want)
