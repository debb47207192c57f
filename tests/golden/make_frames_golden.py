"""Writes tests/golden/frames.npz and solves.npz: the results of the build that
is loaded for the cases of tests/test_gpu_same_results.py.  (The stored ones are
of the build before commit c5c32e3.)  Needs the GPU."""
import sys
from pathlib import Path

import numpy as np

ROOT = Path(__file__).resolve().parents[2]
sys.path[:0] = [str(ROOT / "tests")]

from conftest import load_package  # noqa: E402
import test_gpu_same_results as t  # noqa: E402

if __name__ == "__main__":
    mm = load_package()
    np.savez(t.GOLDEN / "frames.npz", **{k: v for c in t.FRAMES for k, v in t.frames(mm, *c).items()})
    np.savez(t.GOLDEN / "solves.npz", **{k: v for c in t.SOLVES for k, v in t.solve(mm, *c).items()})
