"""Results that users keep: what a graph's whitening and solve gave before the
factorisations and the step were rewritten for speed, they still give.

Nothing in the method fixes the sign of an eigenvector: whitened data stand in
the frame that the FP32 Jacobi leaves, which hangs on every rounding in front of
it (the Cholesky factors, the Gram-Schmidt, the column scalings), and a seeded
Phi stands in that frame.  The first steps of a solve enlarge round-off by their
condition number.  So the stored results (tests/golden/make_frames_golden.py)
are compared as a user sees them, to FP32 round-off, and bit for bit through a
digest where only the last bits show the rounding."""
import hashlib
from pathlib import Path

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
GOLDEN = Path(__file__).resolve().parent / "golden"


def block(mm, rng, zr, zc, k, p_in, p_out):
    nr, nc = len(zr), len(zc)
    m = int(round(p_out * nr * nc))
    rows, cols = [rng.randint(0, nr, m)], [rng.randint(0, nc, m)]
    for c in range(k):
        r, q = np.flatnonzero(zr == c), np.flatnonzero(zc == c)
        i, j = np.nonzero(rng.random_sample((len(r), len(q))) < p_in)
        rows.append(r[i])
        cols.append(q[j])
    key = np.unique(np.concatenate(rows).astype(np.int64) * nc + np.concatenate(cols))
    rp = np.zeros(nr + 1, np.int64)
    np.cumsum(np.bincount(key // nc, minlength=nr), out=rp[1:])
    return mm.CsrBlock(nr, nc, rp, (key % nc).astype(np.int32))


def graph(mm, seed, n, k, p_in, p_out):
    """A block model; RandomState's stream never changes."""
    rng = np.random.RandomState(seed)
    parts = [n // 4 + d for d in (3, -5, 0, 2)]
    z = [rng.randint(0, k, m) for m in parts]
    return mm.Graph([block(mm, rng, z[a], z[b], k, p_in, p_out)
                     for a, b in ((0, 1), (0, 2), (0, 3), (2, 1), (3, 1))], parts)


def digest(*arrays):
    h = hashlib.sha256()
    for a in arrays:
        h.update(np.ascontiguousarray(a).tobytes())
    return np.frombuffer(h.digest(), np.uint8)


def rel(a, b):
    return float(np.linalg.norm(np.asarray(a) - np.asarray(b)) / np.linalg.norm(b))


def frames(mm, k, seed):
    g = graph(mm, 1000 * k + seed, 90 * k if k > 30 else 2200, k, 0.5, 0.004 if k > 30 else 0.01)
    with mm.Pipeline(k=k, alpha0=0.3, seed=seed) as p:
        y = p.upload(g).whiten().whitened()
    return {f"mu_{k}_{seed}": np.stack([np.asarray(y[q + "_mu"], np.float32)
                                        for q in ("Da", "Db", "Dc")]),
            f"digest_{k}_{seed}": digest(*[y[q] for q in ("Da", "Db", "Dc")])}


# frames that another rounding of the Cholesky factors turned
TURNED = [(130, 2), (130, 19), (150, 3), (150, 6), (200, 1), (200, 4)]
# last bits that another order of the Gram-Schmidt's sums changed
BITS_GS = [(100, 0), (100, 8), (130, 1)]
# last bits that column factors of 48 bits changed
BITS_SCALE = [(150, 3), (200, 0)]
FRAMES = sorted(set(TURNED + BITS_GS + BITS_SCALE))


@pytest.mark.parametrize("k,seed", TURNED)
def test_whitening_keeps_its_frame(mm, k, seed):
    with np.load(GOLDEN / "frames.npz") as z:
        want = z[f"mu_{k}_{seed}"]
    assert rel(frames(mm, k, seed)[f"mu_{k}_{seed}"], want) < 2e-5


@pytest.mark.parametrize("k,seed", BITS_GS + BITS_SCALE)
def test_whitening_keeps_its_bits(mm, k, seed):
    with np.load(GOLDEN / "frames.npz") as z:
        want = z[f"digest_{k}_{seed}"]
    assert np.array_equal(frames(mm, k, seed)[f"digest_{k}_{seed}"], want)


def solve(mm, method, precision, k, seed):
    g = graph(mm, 77 + 1000 * k + seed, 2100 + 5 * (seed % 40), k, 0.3, 0.01)
    cfg = dict(stpm_method=getattr(mm, "STPM_" + method), precision=getattr(mm, "PREC_" + precision),
               sweeps=5, minibatch=-(-g.parts[0] // 8), seed=seed, tau=0.2)
    with mm.Pipeline(k=k, alpha0=1.0, **cfg) as p:
        p.upload(g).run()
        lam, pi, phi = p.lam(), p.pi(), p.phi()
    name = f"{method}_{precision}_{k}_{seed}"
    return {"lam_" + name: np.asarray(lam), "digest_" + name: digest(pi, phi)}


# graphs of 2,100 to 2,300 nodes whose lambda another rounding of the k x k step
# or of the contraction moved by 2.6e-5 to 0.6
MOVED = [("ONLINE", "FP32", 5, 1), ("ONLINE", "FP32", 5, 91), ("ONLINE", "FP32", 6, 22),
         ("ONLINE", "FP32", 8, 27), ("ONLINE", "FP32", 12, 19), ("ONLINE", "BF16", 6, 6),
         ("ONLINE", "BF16", 12, 8)]
MOVED += [("ADJOINT", "FP32", 5, 3), ("ADJOINT", "FP32", 8, 29), ("ADJOINT", "FP32", 12, 39),
          ("ADJOINT", "BF16", 6, 1), ("ADJOINT", "BF16", 12, 19)]
SOLVES = MOVED


@pytest.mark.parametrize("method,precision,k,seed", MOVED)
def test_solve_keeps_its_results(mm, method, precision, k, seed):
    name = f"{method}_{precision}_{k}_{seed}"
    got = solve(mm, method, precision, k, seed)
    with np.load(GOLDEN / "solves.npz") as z:
        assert rel(got["lam_" + name], z["lam_" + name]) < 2e-5
        assert np.array_equal(got["digest_" + name], z["digest_" + name])
