"""Reading results takes no device memory: a context that just fitted the GPU
can still be read.  Panels with padding columns (k not a multiple of 4), in
sizes around the staging slots (1 MB, eight of them)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def context(mm, k, nx):
    rng = np.random.default_rng(nx + k)
    y = {n: rng.standard_normal((k, nx)).astype(np.float32) for n in ("Da", "Db", "Dc")}
    mu = {n + "_mu": v.mean(axis=1).astype(np.float64) for n, v in y.items()}
    e = mm.CsrBlock(nx, 1, np.zeros(nx + 1, np.int64), np.zeros(0, np.int32))
    o = mm.CsrBlock(1, 1, np.zeros(2, np.int64), np.zeros(0, np.int32))
    p = mm.Pipeline(k=k, alpha0=1.0)
    p.upload(mm.Graph([e, e, e, o, o], (nx, 1, 1, 1)))
    return p.set_whitened({**{n: v.astype(np.float64) for n, v in y.items()}, **mu}), y


def test_first_get_takes_no_device_memory(mm):
    torch = pytest.importorskip("torch")
    with context(mm, 5, 2000)[0] as p:  # CUDA's own first-use allocations
        p.whitened()
    p, y = context(mm, 75, 150000)
    with p:
        torch.cuda.synchronize()
        before = torch.cuda.mem_get_info()[0]
        got = p.whitened()
        after = torch.cuda.mem_get_info()[0]
    assert before - after < 4 << 20
    assert np.array_equal(got["Da"], y["Da"])


@pytest.mark.parametrize("k,nx", [(1, 1), (3, 70), (6, 5462), (7, 131073), (101, 2521), (101, 10084),
                                  (100, 10486), (33, 60001)])
def test_whitened_rows(mm, k, nx):
    p, y = context(mm, k, nx)
    with p:
        got = p.whitened()
    for n in y:
        assert np.array_equal(got[n], y[n])


@pytest.mark.parametrize("k,nx", [(4, 5000), (8, 100000), (100, 60000)])
def test_whitened_rows_into_old_and_new_pages(mm, k, nx):
    """The same rows whether the buffer's pages were touched (numpy.ones, another
    array's memory used again) or not (a fresh mapping)."""
    import ctypes
    import mmap
    p, y = context(mm, k, nx)
    with p:
        for make in (lambda: np.ones(k * nx, np.float32),
                     lambda: np.frombuffer(mmap.mmap(-1, 4 * k * nx), np.float32)):
            outs = [make() for _ in range(3)]
            for _ in range(2):
                ptr = [o.ctypes.data_as(ctypes.POINTER(ctypes.c_float)) for o in outs]
                p._ck(mm.lib().mmsb_get_whitened(p._h, *ptr, None, None, None))
                for o, n in zip(outs, ("Da", "Db", "Dc")):
                    assert np.array_equal(o.reshape((k, nx), order="F"), y[n])
                    o[:] = 0.0
