"""The calls that a user of this library makes, as cases that can be timed.

A user uploads the five adjacency blocks of a partitioned graph, whitens, runs
the tensor power method (STPM) and unwhitens; or feeds one stage with results
of an earlier run.  Every case goes through the Python mirror of the C ABI,
with host arrays in and out as that ABI has them (pinned where a program that
calls repeatedly would pin them).

Graphs are mixed-membership block models in the shapes of the benchmark and
the tests: four random partitions, Dirichlet(alpha0 / k) memberships, edge
probability p_in inside a community and p_out outside.  Whitened data for the
STPM cases are drawn from the model itself: y = Phi* diag-scaled memberships
plus unit noise, three independent draws.

Which outputs can be compared sets where whole solves are cut: from k of about
ten the online STPM of a sampled graph is decided by round-off (the FP64
iteration itself moves by O(1) under a 1e-7 change of its input), so whole
solves and batches have few communities, and larger sizes run stage by stage
on inputs that determine the result; for the same reason the larger STPM cases
start from a perturbed solution instead of a random frame, from which the order
of many columns hangs on near ties.
"""
import importlib.util
import math
import os
import sys
from pathlib import Path

import numpy as np
import torch

# the graphs of a batch run on streams of their own: read when
# the CUDA context is created
os.environ.setdefault("CUDA_DEVICE_MAX_CONNECTIONS", "32")

_PKG = "fast-detection-of-overlapping-communities-via-online-tensor-methods_gb300"


def _package():
    if "mmsb_gb300" in sys.modules:
        return sys.modules["mmsb_gb300"]
    root = Path.cwd() / _PKG
    spec = importlib.util.spec_from_file_location("mmsb_gb300", root / "__init__.py",
                                                  submodule_search_locations=[str(root)])
    mod = importlib.util.module_from_spec(spec)
    sys.modules["mmsb_gb300"] = mod
    spec.loader.exec_module(mod)
    return mod


def listed():
    return [
        # the smallest whole call: one 4,000-node graph, upload to memberships;
        # launches and latency count
        dict(name="solve_n4000_k5", kind="solve", n=4000, k=5, alpha0=1.0, p_in=0.3, p_out=0.01,
             sweeps=10, minibatch=100),
        # many small graphs in one batched solve
        dict(name="batch16_k4to6", kind="batch", graphs=16, n_lo=2000, n_hi=20000, k_lo=4, k_hi=6,
             alpha0=1.0, p_in=0.3, p_out=0.01, sweeps=5),
        # whitening of a small weighted graph, the size of a batch's larger members
        dict(name="whiten_n20k_k25_weighted", kind="whiten", n=20000, k=25, alpha0=0.5, p_in=0.2,
             p_out=0.002, weighted=True),
        # whitening of the benchmark's graph (n = 200,000, k = 100)
        dict(name="whiten_n200k_k100", kind="whiten", n=200000, k=100, alpha0=0.1, p_in=0.05,
             p_out=5e-4, weighted=False),
        # the largest: panels wider than L2, k above 128
        dict(name="whiten_n600k_k150", kind="whiten", n=600000, k=150, alpha0=0.3, p_in=0.02,
             p_out=2e-5, weighted=False),
        # online STPM, the reference's CPU-runnable schedule: 100 tiny steps
        dict(name="stpm_x1000_k10_b100", kind="stpm", nx=1000, k=10, alpha0=1.0, method="online",
             bf16=False, warm=False, sweeps=10, minibatch=100),
        # online STPM, the benchmark's partition, k and minibatch
        dict(name="stpm_x50k_k100_b4096", kind="stpm", nx=50000, k=100, alpha0=0.1,
             method="online", bf16=False, warm=True, sweeps=5, minibatch=4096),
        # online STPM at the largest k in use
        dict(name="stpm_x65k_k200_b8192", kind="stpm", nx=65000, k=200, alpha0=0.3,
             method="online", bf16=False, warm=True, sweeps=5, minibatch=8192),
        # adjoint STPM with BF16 data, odd sizes
        dict(name="stpm_x30011_k75_adj_bf16", kind="stpm", nx=30011, k=75, alpha0=0.3,
             method="adjoint", bf16=True, warm=True, sweeps=4, minibatch=2048),
        # the default method: full-batch power iteration
        dict(name="power_x10k_k33", kind="power", nx=10000, k=33, alpha0=0.5, iters=150),
        # the loss of one minibatch and its gradient
        dict(name="loss_x8192_k100", kind="loss", nx=8192, k=100, alpha0=1.0),
        # unwhitening and normalisation of the benchmark's graph
        dict(name="post_n200k_k100", kind="post", n=200000, k=100, alpha0=0.1, p_in=0.05,
             p_out=5e-4),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["solve", "batch", "whiten", "whiten", "stpm", "stpm", "stpm", "power",
                       "loss", "post"])
    if kind == "solve":
        n = _log(rng, 2000, 30000)
        return dict(kind=kind, n=n, k=rng.randint(4, 6), alpha0=round(rng.uniform(0.3, 1.0), 2),
                    p_in=round(rng.uniform(0.2, 0.3), 3), p_out=0.01, sweeps=rng.randint(6, 12),
                    minibatch=max(64, n // rng.randint(36, 60)))
    if kind == "batch":
        return dict(kind=kind, graphs=rng.randint(5, 16), n_lo=2000, n_hi=_log(rng, 4000, 20000),
                    k_lo=4, k_hi=6, alpha0=round(rng.uniform(0.5, 1.0), 2), p_in=0.3, p_out=0.01,
                    sweeps=rng.randint(4, 6))
    if kind in ("whiten", "post"):
        n = _log(rng, 8000, 300000)
        k = rng.randint(10, max(12, min(128, n // 500)))
        # mean degree 40 to 160, three quarters of it inside the communities
        deg = rng.uniform(40.0, 160.0)
        c = dict(kind=kind, n=n, k=k, alpha0=round(rng.uniform(0.1, 0.6), 2),
                 p_in=min(0.5, 0.75 * deg * k / n), p_out=0.25 * deg / n)
        if kind == "whiten":
            c["weighted"] = rng.random() < 0.3
        return c
    if kind == "stpm":
        nx, k = _log(rng, 1000, 65000), rng.choice([rng.randint(6, 40), rng.randint(41, 112),
                                                    rng.randint(113, 204)])
        nx = max(nx, 200 * k)
        b = max(40 * k, _log(rng, 64, 16384))
        per = -(-nx // b)
        bf16 = rng.random() < 0.4
        # enough steps that the iterate has settled: a few steps from the
        # start it still carries the round-off of ill-conditioned first steps
        return dict(kind=kind, nx=nx, k=k, alpha0=round(rng.uniform(0.1, 1.0), 2),
                    method=rng.choice(["online", "online", "adjoint"]), bf16=bf16,
                    warm=bf16 or k > 48,
                    sweeps=max(3, -(-50 // per)), minibatch=b)
    if kind == "power":
        return dict(kind=kind, nx=_log(rng, 1000, 20000), k=rng.randint(5, 64),
                    alpha0=round(rng.uniform(0.1, 1.0), 2), iters=rng.randint(100, 160))
    return dict(kind=kind, nx=_log(rng, 1000, 30000), k=rng.randint(10, 120),
                alpha0=round(rng.uniform(0.1, 1.0), 2))


# ---- inputs -------------------------------------------------------------------


def _host(t):
    """A pinned host copy as numpy (the array keeps the memory alive)."""
    h = torch.empty(t.shape, dtype=t.dtype, pin_memory=True)
    h.copy_(t)
    return h.numpy()


def _memberships(gen, n, k, alpha0):
    a = torch.full((n, k), alpha0 / k, device="cuda", dtype=torch.float32)
    # Gamma(a) = Gamma(a + 1) U^(1/a), in logarithms: a is far below one
    g = torch._standard_gamma(a + 1.0, generator=gen).log_()
    u = torch.rand((n, k), device="cuda", generator=gen).clamp_min_(1e-30).log_()
    return torch.softmax(g + u / a, dim=1)


def _block(mm, gen, pr, pc, p_in, p_out, weighted):
    """CSR block of edges between the nodes of two partitions."""
    nr, nc, k = pr.shape[0], pc.shape[0], pr.shape[1]

    def poisson(mean):
        return int(torch.poisson(torch.tensor([float(mean)], device="cuda"), generator=gen).item())

    m0 = poisson(p_out * nr * nc)
    rows = [torch.randint(nr, (m0,), device="cuda", generator=gen)]
    cols = [torch.randint(nc, (m0,), device="cuda", generator=gen)]
    # inside: the community with weight (mass of rows) x (mass of columns), then
    # each end with its membership weight
    cr, cc = pr.t().double().reshape(-1).cumsum(0), pc.t().double().reshape(-1).cumsum(0)
    er = torch.cat([cr.new_zeros(1), cr[nr - 1::nr]])
    ec = torch.cat([cc.new_zeros(1), cc[nc - 1::nc]])
    mass = (er[1:] - er[:-1]) * (ec[1:] - ec[:-1])
    m1 = poisson((p_in - p_out) * float(mass.sum()))
    cm = mass.cumsum(0)
    pick = torch.rand(m1, device="cuda", dtype=torch.float64, generator=gen) * cm[-1]
    com = torch.searchsorted(cm, pick).clamp_(max=k - 1)
    for cum, edge, n, out in ((cr, er, nr, rows), (cc, ec, nc, cols)):
        u = torch.rand(m1, device="cuda", dtype=torch.float64, generator=gen)
        at = torch.searchsorted(cum, edge[com] + u * (edge[com + 1] - edge[com]))
        out.append((at - com * n).clamp_(0, n - 1))
    key = torch.unique(torch.cat(rows) * nc + torch.cat(cols))
    ri, ci = key // nc, (key % nc).int()
    rp = torch.zeros(nr + 1, device="cuda", dtype=torch.int64)
    rp[1:] = torch.bincount(ri, minlength=nr).cumsum(0)
    val = None
    if weighted:
        val = _host(torch.rand(ci.shape[0], device="cuda", generator=gen) * 1.5 + 0.5)
    return mm.CsrBlock(nr, nc, _host(rp), _host(ci), val)


def _graph(mm, seed, n, k, alpha0, p_in, p_out, weighted=False, with_pi=False):
    gen = torch.Generator("cuda").manual_seed(int(seed) * 1000003 + n * 31 + k)
    # uneven partitions that depend on the sizes only, as a file's would
    part = np.random.default_rng(n + k).multinomial(n, [0.25] * 4).tolist()
    pi = [_memberships(gen, m, k, alpha0) for m in part]
    ends = ((0, 1), (0, 2), (0, 3), (2, 1), (3, 1))  # X-A, X-B, X-C, B-A, C-A
    g = mm.Graph([_block(mm, gen, pi[r], pi[c], p_in, p_out, weighted) for r, c in ends], part)
    return (g, pi, gen) if with_pi else g


def _orthonormal(gen, k):
    q, r = torch.linalg.qr(torch.randn(k, k, generator=gen, dtype=torch.float64))
    return q * torch.sign(torch.diagonal(r))


def _whitened(case, seed):
    """Whitened data of the model: y_q = sqrt(k (a0 + 1)) Phi* pi + noise, their
    means, the components Phi* and an orthonormal start: random, or ("warm") a
    perturbed Phi*, as a run that goes on from an earlier solve has it."""
    nx, k, a0 = case["nx"], case["k"], case["alpha0"]
    cpu = torch.Generator().manual_seed(int(seed) * 7919 + nx * 13 + k)
    gen = torch.Generator("cuda").manual_seed(int(seed) * 104729 + nx * 17 + k)
    comp, start = _orthonormal(cpu, k), _orthonormal(cpu, k)
    if case.get("warm"):
        start = comp + 0.5 / math.sqrt(k) * torch.randn(k, k, generator=cpu, dtype=torch.float64)
        q, r = torch.linalg.qr(start)
        start = q * torch.sign(torch.diagonal(r))
    h = _memberships(gen, nx, k, a0).double() @ comp.cuda().t() * math.sqrt(k * (a0 + 1.0))
    y = [(h + torch.randn((nx, k), device="cuda", dtype=torch.float64, generator=gen)).float()
         for _ in range(3)]
    mu = [v.double().mean(0).cpu().numpy() for v in y]
    return y, mu, comp.numpy(), start.float().double().numpy()


def _stage(mm, case, seed, **cfg):
    """A context that holds whitened data (its graph has the X nodes only in
    number: the STPM does not read it)."""
    nx = case["nx"]
    y, mu, comp, start = _whitened(case, seed)
    e = mm.CsrBlock(nx, 1, np.zeros(nx + 1, np.int64), np.zeros(0, np.int32))
    o = mm.CsrBlock(1, 1, np.zeros(2, np.int64), np.zeros(0, np.int32))
    p = mm.Pipeline(k=case["k"], alpha0=case["alpha0"], **cfg)
    p.upload(mm.Graph([e, e, e, o, o], (nx, 1, 1, 1)))
    p.set_whitened(dict(Da=y[0].double().cpu().numpy().T, Db=y[1].double().cpu().numpy().T,
                        Dc=y[2].double().cpu().numpy().T, Da_mu=mu[0], Db_mu=mu[1], Dc_mu=mu[2]))
    return p, comp, start


def prepare(case, seed):
    mm = _package()
    kind = case["kind"]
    st = dict(kind=kind, mm=mm)
    if kind == "solve":
        g = _graph(mm, seed, case["n"], case["k"], case["alpha0"], case["p_in"], case["p_out"])
        st.update(graph=g, p=mm.Pipeline(k=case["k"], alpha0=case["alpha0"],
                                         stpm_method=mm.STPM_ONLINE, sweeps=case["sweeps"],
                                         minibatch=case["minibatch"], seed=seed & 0xffff, tau=0.2),
                  pi=_host(torch.zeros((case["n"], case["k"]))).T)
    elif kind == "batch":
        m = case["graphs"]
        rng = np.random.default_rng(m + case["n_hi"])  # uneven, the same for every seed
        ns = np.exp(rng.uniform(np.log(case["n_lo"]), np.log(case["n_hi"]), m)).astype(int)
        ks = rng.integers(case["k_lo"], case["k_hi"] + 1, m)
        gs = [_graph(mm, seed * 64 + i, int(n), int(k), case["alpha0"], case["p_in"],
                     case["p_out"]) for i, (n, k) in enumerate(zip(ns, ks))]
        b = mm.Batch(ks, [case["alpha0"]] * m, [-(-g.parts[0] // 8) for g in gs],
                     stpm_method=mm.STPM_ONLINE, sweeps=case["sweeps"], seed=seed & 0xffff,
                     tau=0.2)
        for i, g in enumerate(gs):
            b.upload(i, g)
        st.update(b=b, pi=[_host(torch.zeros((int(n), int(k)))).T for n, k in zip(ns, ks)])
    elif kind == "whiten":
        g = _graph(mm, seed, case["n"], case["k"], case["alpha0"], case["p_in"], case["p_out"],
                   case["weighted"])
        st["p"] = mm.Pipeline(k=case["k"], alpha0=case["alpha0"], datatype=int(case["weighted"]),
                              seed=seed & 0xffff)
        st["p"].upload(g)
    elif kind == "stpm":
        st["p"], _, st["phi0"] = _stage(
            mm, case, seed, stpm_method=getattr(mm, "STPM_" + case["method"].upper()),
            precision=mm.PREC_BF16 if case["bf16"] else mm.PREC_FP32, sweeps=case["sweeps"],
            minibatch=case["minibatch"])
    elif kind == "power":
        # tol = 0: exactly iters + 1 iterations, the same work for every seed
        st["p"], _, st["phi0"] = _stage(mm, case, seed, stpm_method=mm.STPM_BATCH_POWER,
                                        min_iter=case["iters"], max_iter=case["iters"], tol=0.0)
    elif kind == "loss":
        # an iterate half way to the components
        st["p"], comp, start = _stage(mm, case, seed, theta=1.0)
        st["phi"] = (0.7 * comp + 0.3 * start).astype(np.float32).astype(np.float64)
    else:
        x = _post_inputs(mm, case, seed)
        p = mm.Pipeline(k=case["k"], alpha0=case["alpha0"], tau=0.1)
        p.upload(x["graph"])
        p.set_whitening({n: v.double().cpu().numpy() if n not in ("Zb2", "Zc2")
                         else v.double().cpu().numpy().T for n, v in x["wh"].items()})
        p.set_phi_lambda(x["phi"], x["lam"])
        st.update(p=p, pi=_host(torch.zeros((case["n"], case["k"]))).T)
    return st


def _post_inputs(mm, case, seed):
    """A whitening in the model's own frame: W and the pair factors are the
    memberships of their partitions times Phi*^T, slightly perturbed, as a
    converged run has them; memberships come out of the neighbourhoods."""
    n, k = case["n"], case["k"]
    g, pi, gen = _graph(mm, seed, n, k, case["alpha0"], case["p_in"], case["p_out"], with_pi=True)
    comp = _orthonormal(torch.Generator().manual_seed(int(seed) * 31 + k), k)
    q = comp.float().cuda().t()

    def panel(m):
        v = m @ q
        return v * (1.0 + 0.05 * torch.randn(v.shape, device="cuda", generator=gen))

    wh = dict(W=panel(pi[1]), Zb1=panel(pi[1]) * (k / pi[1].shape[0]), Zb2=panel(pi[2]),
              Zc1=panel(pi[1]) * (k / pi[1].shape[0]), Zc2=panel(pi[3]),
              mu_a=pi[1].mean(1), mu_b=pi[2].mean(1), mu_c=pi[3].mean(1))
    lam = np.linspace(1.0, 2.0, k) * math.sqrt(k)
    return dict(graph=g, wh=wh, phi=comp.float().double().numpy(), lam=lam)


# ---- the calls ------------------------------------------------------------------
#
# lambda, Phi, the whitened means, the loss and its gradient are FP32 results
# that the getters widen to FP64; they are returned in FP32.


def run(st):
    kind = st["kind"]
    if kind == "solve":
        p = st["p"].upload(st["graph"]).run()
        return dict(pi=p.pi(out=st["pi"]), lam=p.lam().astype(np.float32))
    if kind == "batch":
        b = st["b"].run()
        g = [b.graph(i) for i in range(len(b))]
        return dict(pi=[p.pi(out=o) for p, o in zip(g, st["pi"])],
                    lam=[p.lam().astype(np.float32) for p in g])
    p = st["p"]
    if kind == "whiten":
        return {n: v.astype(np.float32, copy=False) for n, v in p.whiten().whitened().items()}
    if kind in ("stpm", "power"):
        p.stpm(st["phi0"])
        return dict(phi=p.phi().astype(np.float32), lam=p.lam().astype(np.float32))
    if kind == "loss":
        return dict(loss=np.float32(p.loss(st["phi"])),
                    grad=p.loss_grad(st["phi"]).astype(np.float32))
    return p.postproc().pi(out=st["pi"])


# ---- least work -----------------------------------------------------------------


def _nnz(n, k, p_in, p_out):
    # five of the pairs of four equal partitions; memberships nearly pure
    return 5.0 * (n / 4.0) ** 2 * (p_out + (p_in - p_out) / k)


def _whiten_work(n, k, p_in, p_out, weighted=False):
    nq, e = n / 4.0, _nnz(n, k, p_in, p_out) / 5.0
    p = 2.0 * k
    # per side: 4 products with p columns and 2 with k; then 4 with k for the
    # pair factors and the core, 3 for the whitened data
    flops = 2.0 * e * (2 * (4 * p + 2 * k) + 7 * k)
    # Grams and panel products of the three Nystrom steps
    flops += 2.0 * nq * (2 * (3 * p * p + p * k) + 3 * k * k + 2 * k * p + 5 * k * k)
    byts = 3 * (e * (8 if weighted else 4) + 8 * nq) + 3 * 4.0 * nq * k
    return byts, flops


def work(case):
    kind, k = case["kind"], float(case.get("k", 0))
    if kind in ("solve", "whiten"):
        b, f = _whiten_work(case["n"], k, case["p_in"], case["p_out"], case.get("weighted", False))
        if kind == "solve":
            nx, e = case["n"] / 4.0, _nnz(case["n"], k, case["p_in"], case["p_out"])
            f += case["sweeps"] * nx * 6 * k * k + 2 * k * e
            b += 8 * e + 4.0 * case["n"] * k
        return dict(bytes=b, flops=f)
    if kind == "batch":
        n, k = math.sqrt(case["n_lo"] * case["n_hi"]), (case["k_lo"] + case["k_hi"]) / 2.0
        b, f = _whiten_work(n, k, case["p_in"], case["p_out"])
        e = _nnz(n, k, case["p_in"], case["p_out"])
        f += case["sweeps"] * n / 4.0 * 6 * k * k + 2 * k * e
        return dict(bytes=case["graphs"] * (b + 4.0 * n * k + 4 * e), flops=case["graphs"] * f)
    if kind == "stpm":
        products = 12.0 if case["method"] == "adjoint" else 6.0
        steps = case["sweeps"] * -(-case["nx"] // case["minibatch"])
        size = 2.0 if case["bf16"] else 4.0
        # y of a sweep stays in L2 or is read again: counted once
        return dict(bytes=3 * size * case["nx"] * k + 8 * k * k,
                    flops=case["sweeps"] * case["nx"] * products * k * k + steps * 10 * k ** 3)
    if kind == "power":
        return dict(bytes=12.0 * case["nx"] * k + 8 * k * k,
                    flops=(case["iters"] + 1.0) * case["nx"] * 6 * k * k)
    if kind == "loss":
        return dict(bytes=12.0 * case["nx"] * k + 8 * k * k,
                    flops=case["nx"] * 18 * k * k + 6 * k ** 3)
    n, e = case["n"], _nnz(case["n"], k, case["p_in"], case["p_out"])
    return dict(bytes=4 * e * 0.8 + 8.0 * n + 4.0 * n * k + 12.0 * n / 4 * k,
                flops=2 * k * e * 0.8 + 6 * (n / 4) * k * k)


# ---- 64 bits ---------------------------------------------------------------------


def _coeffs(a0):
    return (a0 + 1.0) * (a0 + 2.0) / 2.0, a0 * a0, -a0 * (a0 + 1.0) / 2.0


def _grad(phi, y, mu, p0, p1, p2):
    """Column i: mean over the nodes of T(I, phi_i, phi_i)'s terms, y = (y1, y2, y3)."""
    z1, z2 = y[0] @ phi, y[1] @ phi
    m1, m2 = mu[0] @ phi, mu[1] @ phi
    c = p0 * z1 * z2 + p2 * (z1 * m2 + m1 * z2)
    return y[2].T @ c / len(z1) + torch.outer(mu[2], p1 * m1 * m2 + p2 * (z1 * z2).mean(0))


def _adjoint(phi, y, mu, p0, p1, p2):
    a, b, c = ([y[i], y[j], y[q]] for i, j, q in ((0, 1, 2), (0, 2, 1), (1, 2, 0)))
    order = ((0, 1, 2), (0, 2, 1), (1, 2, 0))
    return sum(_grad(phi, v, [mu[i] for i in o], p0, p1, p2) for v, o in zip((a, b, c), order))


def _qr(x):
    q, r = torch.linalg.qr(x)
    return q * torch.sign(torch.diagonal(r))


def exact(case, seed):
    kind = case["kind"]
    if kind in ("solve", "batch", "whiten"):
        return None  # columns of W have a sign and, close to one another, a rotation of their own
    if kind == "post":
        return _exact_post(case, seed)
    y, mu, comp, start = _whitened(case, seed)
    # on the GPU in 64 bits, a chunk of the nodes at a time being the minibatch
    y = [v.double() for v in y]
    mu = [torch.from_numpy(m).cuda() for m in mu]
    co = _coeffs(case["alpha0"])
    if kind == "loss":
        phi = (0.7 * comp + 0.3 * start).astype(np.float32).astype(np.float64)
        phi = torch.from_numpy(phi).cuda()
        g = _grad(phi, y, mu, *co)
        s = phi.T @ phi
        # theta = 1; the cubic form is phi_i . G_i up to the mean terms of the third slot
        z = [v @ phi for v in y]
        m = [v @ phi for v in mu]
        that = (co[0] * z[0] * z[1] * z[2] + co[2] * (z[0] * z[1] * m[2] + z[0] * m[1] * z[2]
                                                      + m[0] * z[1] * z[2])).mean(0)
        that = that + co[1] * m[0] * m[1] * m[2]
        assert torch.allclose(that, (phi * g).sum(0), rtol=1e-8, atol=1e-8)
        loss = (s ** 3).sum() - 2.0 * that.sum()
        grad = 6.0 * phi @ (s * s) - 2.0 * _adjoint(phi, y, mu, *co)
        return dict(loss=loss.cpu().numpy(), grad=grad.cpu().numpy())
    phi = torch.from_numpy(start).cuda()
    if kind == "power":
        order = (1, 2, 0)
        yy, mm_ = [y[i] for i in order], [mu[i] for i in order]
        for _ in range(case["iters"] + 1):
            new = _grad(phi, yy, mm_, *co)
            norm = new.norm(dim=0)
            phi = new / norm
        return dict(phi=phi.cpu().numpy(), lam=(norm ** 3).cpu().numpy())
    t, b = 0, case["minibatch"]
    for _ in range(case["sweeps"]):
        for x0 in range(0, case["nx"], b):
            part = [v[x0:x0 + b] for v in y]
            o = 1.5 * phi @ ((phi.T @ phi) ** 2)
            if case["method"] == "adjoint":
                step = o - _adjoint(phi, part, mu, *co)
            else:
                step = o - 3.0 * _grad(phi, part, mu, *co)
            phi = _qr(phi - step / (1.0 + t))
            t += 1
    lam = (phi * _grad(phi, y, mu, *co)).sum(0)
    sign = torch.where(lam < 0, -1.0, 1.0)
    return dict(phi=(phi * sign).cpu().numpy(), lam=(lam * sign).cpu().numpy())


def _exact_post(case, seed):
    x = _post_inputs(_package(), case, seed)
    wh = {n: v.double() for n, v in x["wh"].items()}
    pa = wh["W"] @ (torch.from_numpy(x["phi"]).cuda() / torch.from_numpy(x["lam"]).cuda())
    pa2 = wh["Zb2"] @ (wh["Zb1"].T @ pa)

    def product(block, panel, transpose=False):
        rows = torch.repeat_interleave(torch.arange(block.n_rows, device="cuda"),
                                       torch.from_numpy(np.diff(block.row_ptr)).cuda())
        cols = torch.from_numpy(block.col_idx).cuda().long()
        if transpose:
            rows, cols = cols, rows
        out = torch.zeros((block.n_cols if transpose else block.n_rows, panel.shape[1]),
                          device="cuda", dtype=torch.float64)
        for at in range(0, len(rows), 1 << 20):
            out.index_add_(0, rows[at:at + (1 << 20)], panel[cols[at:at + (1 << 20)]])
        return out

    blocks = x["graph"].blocks
    raw = torch.cat([product(blocks[0], pa), product(blocks[3], pa2, True),
                     product(blocks[3], pa), product(blocks[4], pa)])
    pos, neg = raw.clamp_min(0).sum(1, keepdim=True), raw.clamp_max(0).sum(1, keepdim=True).abs()
    flip = pos < neg
    out = torch.where(flip, -raw / neg, raw / torch.where(pos == 0, torch.ones_like(pos), pos))
    return out.clamp_min(0).T.cpu().numpy()
