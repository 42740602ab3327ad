"""The work that users of this library have it do, as cases that can be timed
and compared: each goes through the package's public calls, over the sizes of
the repository's configurations, tests and benchmark (workloads.py, bench.py,
bench_extra.py) and odd sizes between them.

A case names its path:

  solve      paralanczos_b200.solve, uniform k, device tensors (the hot path)
  solve_all  the same with want_all (every eigenvalue and the determinant)
  csr        solve with CSR offsets: uneven k in one binned launch
  host       solve_host: numpy buffers in and out
  dropin     calculate_subeigs3, the entry point of C and MATLAB callers: FP64
             host matrix, every eigenvalue
  gram       GramFrame.solve: A[S,S] formed on the fly from the frame
  blocks     GramFrame.blocks: the Gram blocks themselves
  serve      Server: a burst of requests of different k, size and matrix

``prepare`` makes the inputs from the seed on the GPU (host arrays where the
call takes host arrays) with torch alone; ``run`` is one call and its outputs;
``exact`` is LAPACK in FP64 on the same submatrices.
"""
from __future__ import annotations

import concurrent.futures as cf
import math

import numpy as np
import torch

from paralanczos_b200 import api as pl

# The uneven stream's k values; a set has k with probability ~ 1/k.
KVALUES = (8, 16, 24, 32, 48, 64, 96, 128, 192, 256)


def listed():
    return [
        # one short call inside a host loop: launch and dependency latency
        dict(name="small_k16", path="solve", kind="gauss", m=128, n=512, k=16, nsets=256),
        # the reference's own entry point on the small configuration: 10,000
        # sets of 16 columns, FP64 host matrix, every eigenvalue
        dict(name="dropin_k16", path="dropin", kind="gauss", m=128, n=512, k=16, nsets=10_000),
        # host buffers end to end at an odd k
        dict(name="host_k33", path="host", kind="rademacher", m=1024, n=2048, k=33, nsets=30_000),
        # the headline: 1,000,000 sets of 64 columns of a 1024 x 4096 frame
        dict(name="solve_k64", path="solve", kind="gauss", m=1024, n=4096, k=64, nsets=1_000_000),
        # every eigenvalue and the determinant (interior statistics), odd k and n
        dict(name="all_k60", path="solve_all", kind="gauss", m=1024, n=3001, k=60, nsets=50_000),
        # one batch with uneven k (a RIP study over several sparsity levels)
        dict(name="csr_mixed", path="csr", kind="gauss", m=1024, n=4096, nsets=100_000),
        # one SM per set, ragged k, correlated columns
        dict(name="solve_k200", path="solve", kind="corr", m=1024, n=4096, k=200, nsets=3_000),
        # the largest supported sets
        dict(name="solve_k512", path="solve", kind="gauss", m=1024, n=4096, k=512, nsets=600),
        # frames too wide for a materialised A: blocks on the tensor cores
        dict(name="gram_k128", path="gram", kind="rademacher", m=2048, n=16384, k=128, nsets=20_000),
        dict(name="blocks_k50", path="blocks", kind="gauss", m=1024, n=8192, k=50, nsets=20_000),
        # a burst of requests as a service gets them
        dict(name="serve_burst", path="serve", kind="gauss", m=1024, n=4096, requests=12, kmin=8, kmax=512,
             maxsets=400),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _most(k, scale):
    """Most sets of a drawn case: the headline's work at k = 64, fewer for
    larger k (whose sets cost more per operation)."""
    return max(64, int(scale * min(1.0, (64.0 / k) ** 4)))


def draw(rng):
    path = rng.choice(["solve", "solve", "solve", "solve_all", "csr", "host", "dropin", "gram", "blocks", "serve"])
    kind = rng.choice(["gauss", "rademacher", "corr"])
    m = rng.choice([512, 1024, 2048])
    n = rng.randint(m, 4 * m)
    if path == "solve":
        k = _log_int(rng, 4, min(512, m // 2))
        return dict(path=path, kind=kind, m=m, n=n, k=k, nsets=_log_int(rng, 1, _most(k, 1_000_000)))
    if path == "solve_all":
        k = _log_int(rng, 4, 128)
        return dict(path=path, kind=kind, m=m, n=n, k=k, nsets=_log_int(rng, 1, _most(k, 100_000)))
    if path == "csr":
        return dict(path=path, kind=kind, m=1024, n=rng.randint(1024, 4096), nsets=_log_int(rng, 100, 100_000))
    if path == "host":
        k = _log_int(rng, 4, 128)
        return dict(path=path, kind=kind, m=m, n=min(n, 4096), k=k, nsets=_log_int(rng, 10, _most(k, 100_000)))
    if path == "dropin":
        # the reference's rules: k % 4 == 0 and nsets * k % 32 == 0
        k = 4 * rng.randint(1, 16)
        return dict(path=path, kind=kind, m=512, n=rng.randint(256, 1024), k=k,
                    nsets=8 * _log_int(rng, 2, _most(k, 2_500)))
    if path in ("gram", "blocks"):
        k = _log_int(rng, 8, 128)
        return dict(path=path, kind=kind, m=m, n=rng.randint(m, 8192), k=k, nsets=_log_int(rng, 10, 20_000))
    kmax = rng.randint(64, 512)
    return dict(path=path, kind=kind, m=1024, n=rng.randint(1024, 4096), requests=rng.randint(2, 12),
                kmin=8, kmax=kmax, maxsets=rng.randint(20, 400))


# --------------------------------------------------------------------------- inputs


def _frame(kind, m, n, gen):
    """FP32 frame (m x n): N(0, 1/m), Rademacher +-1/sqrt(m), or Gaussian with
    0.3 of its neighbours mixed into every column."""
    if kind == "rademacher":
        P = (torch.randint(0, 2, (m, n), generator=gen, device="cuda").double() * 2 - 1) / math.sqrt(m)
    else:
        P = torch.randn((m, n), generator=gen, device="cuda", dtype=torch.float64) / math.sqrt(m)
        if kind == "corr":
            Q = P.clone()
            Q[:, 1:] += 0.3 * P[:, :-1]
            Q[:, :-1] += 0.3 * P[:, 1:]
            P = Q
    return P.float()


def _gram64(Phi):
    P = Phi.double()
    G = P.T @ P
    return (G + G.T) / 2


def _sets(nsets, n, k, gen):
    """(nsets, k) int64 on the GPU: k distinct values of [0, n) per row."""
    idx = torch.randint(0, n, (nsets, k), generator=gen, device="cuda")
    while True:
        s, order = torch.sort(idx, dim=1)
        dup = torch.zeros_like(s, dtype=torch.bool)
        dup[:, 1:] = s[:, 1:] == s[:, :-1]
        rows = dup.any(1).nonzero().squeeze(1)
        if rows.numel() == 0:
            return idx
        sub = torch.zeros((rows.numel(), k), dtype=torch.bool, device="cuda")
        sub.scatter_(1, order[rows], dup[rows])
        new = torch.randint(0, n, sub.shape, generator=gen, device="cuda")
        idx[rows] = torch.where(sub, new, idx[rows])


def _stream(nsets, n, gen):
    """CSR sets with k of KVALUES, P ~ 1/k: (offsets int64, idx int32)."""
    w = torch.tensor([1.0 / k for k in KVALUES], device="cuda")
    which = torch.multinomial(w, nsets, replacement=True, generator=gen)
    ks = torch.tensor(KVALUES, device="cuda")[which]
    offsets = torch.zeros(nsets + 1, dtype=torch.int64, device="cuda")
    offsets[1:] = torch.cumsum(ks, 0)
    idx = torch.empty(int(offsets[-1]), dtype=torch.int32, device="cuda")
    for i, k in enumerate(KVALUES):
        at = offsets[:-1][which == i]
        if at.numel():
            idx[at[:, None] + torch.arange(k, device="cuda")] = _sets(at.numel(), n, k, gen).int()
    return offsets, idx


def _burst(case):
    """(k, sets) of each request: k spread evenly over its range, sizes over
    their logarithm (the serving workload's distributions), in a mixed order
    that is part of the case."""
    R, k0, k1 = case["requests"], case["kmin"], case["kmax"]
    out = []
    for i in range(R):
        u, v = (i * 0.618034 + 0.3) % 1.0, (i * 0.754878 + 0.5) % 1.0
        out.append((k0 + int(u * (k1 - k0 + 1)), max(1, round(math.exp(v * math.log(case["maxsets"]))))))
    return out


def _inputs(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    Phi = _frame(case["kind"], case["m"], case["n"], gen)
    path, n = case["path"], case["n"]
    if path == "csr":
        offsets, idx = _stream(case["nsets"], n, gen)
        return dict(Phi=Phi, offsets=offsets, idx=idx)
    if path == "serve":
        reqs = [(i % 2, k, _sets(ns, n, k, gen).int().reshape(-1)) for i, (k, ns) in enumerate(_burst(case))]
        other = _frame("rademacher", case["m"], n, gen)
        return dict(Phi=Phi, other=other, reqs=reqs)
    return dict(Phi=Phi, idx=_sets(case["nsets"], n, case["k"], gen).int().reshape(-1))


class _Serving:
    """A running server with its matrices resident, and the burst to send."""

    def __init__(self, mats, reqs):
        self.server = pl.Server(budget_bytes=1 << 30, host_pool_bytes=1 << 26)
        self.ids = [self.server.add_matrix(A) for A in mats]
        self.reqs = [(self.ids[i], k, idx.cpu().numpy()) for i, k, idx in reqs]


def prepare(case, seed):
    x = _inputs(case, seed)
    path = case["path"]
    st = dict(path=path, k=case.get("k"))
    if path in ("gram", "blocks"):
        st.update(frame=pl.GramFrame(x["Phi"]), idx=x["idx"])
    elif path == "serve":
        st["serving"] = _Serving([_gram64(x["Phi"]).float(), _gram64(x["other"]).float()], x["reqs"])
    elif path == "dropin":
        total = case["nsets"] * case["k"]
        st.update(mat=_gram64(x["Phi"]).cpu().numpy(), n=case["n"], total=total, idx=x["idx"].cpu().numpy(),
                  eig=np.zeros(total), det=np.zeros(case["nsets"]))
    elif path == "host":
        st.update(A=_gram64(x["Phi"]).float().cpu().numpy(), idx=x["idx"].cpu().numpy())
    else:
        st.update(A=_gram64(x["Phi"]).float(), idx=x["idx"], offsets=x.get("offsets"))
    return st


# --------------------------------------------------------------------------- one pass


def run(st):
    path = st["path"]
    if path == "csr":
        return pl.solve(st["A"], st["idx"], offsets=st["offsets"])
    if path == "solve":
        return pl.solve(st["A"], st["idx"], k=st["k"])
    if path == "solve_all":
        return pl.solve(st["A"], st["idx"], k=st["k"], want_all=True)
    if path == "host":
        return pl.solve_host(st["A"], st["idx"], k=st["k"])
    if path == "gram":
        return st["frame"].solve(st["idx"], st["k"])
    if path == "blocks":
        return st["frame"].blocks(st["idx"], st["k"])
    if path == "dropin":
        rc = pl.calculate_subeigs3(st["mat"], st["total"], st["n"], st["eig"], st["det"], st["idx"], st["k"])
        return dict(rc=rc, eig=st["eig"], det=st["det"])
    s = st["serving"]
    ids = [s.server.submit(m, idx, k) for m, k, idx in s.reqs]
    out = []
    for rid, (_, k, idx) in zip(ids, s.reqs):
        r = s.server.wait(rid, len(idx) // k)
        out.append({name: r[name] for name in ("lmin", "lmax", "delta", "err")})
    return out


# --------------------------------------------------------------------------- cost and truth


def _spans(case):
    """[(k, number of sets)] of one pass (expected counts for random k)."""
    if case["path"] == "csr":
        tot = sum(1.0 / k for k in KVALUES)
        return [(k, case["nsets"] / k / tot) for k in KVALUES]
    if case["path"] == "serve":
        return _burst(case)
    return [(case["k"], case["nsets"])]


def work(case):
    """Lanczos with full reorthogonalisation takes 4 k^3 flops per set, a Gram
    block 2 m k^2.  Bytes: the indices and the matrix (or frame) once, the
    outputs once."""
    path, n, m = case["path"], case["n"], case["m"]
    flops = nbytes = 0.0
    for k, ns in _spans(case):
        nbytes += ns * 4 * k
        if path == "blocks":
            flops += ns * 2.0 * m * k * k
            nbytes += ns * (4 * k * k + 4)
            continue
        flops += ns * 4.0 * k ** 3
        if path == "gram":
            flops += ns * 2.0 * m * k * k
        nbytes += ns * 28
        if path in ("solve_all", "dropin"):
            nbytes += ns * (8 * k + 8)
    if path in ("gram", "blocks"):
        nbytes += 4.0 * m * n
    elif path == "dropin":
        nbytes += 8.0 * n * n
    else:
        nbytes += 4.0 * n * n * (2 if path == "serve" else 1)
    return dict(bytes=nbytes, flops=flops)


def _eigs(blocks):
    """Ascending eigenvalues of (ns, k, k) FP64 blocks (LAPACK, several threads)."""
    b = blocks.cpu().numpy()
    parts = np.array_split(np.arange(len(b)), min(len(b), 64))
    with cf.ThreadPoolExecutor(8) as ex:
        return np.concatenate(list(ex.map(lambda p: np.linalg.eigvalsh(b[p]), parts)))


def _submatrix_eigs(A, idx, k):
    S = idx.reshape(-1, k).long()
    out = []
    for c in torch.split(S, max(1, (1 << 26) // (k * k))):
        out.append(_eigs(A[c[:, :, None], c[:, None, :]].double()))
    return np.concatenate(out)


def _gram_blocks(Phi, idx, k):
    P = Phi.double().T.contiguous()
    for c in torch.split(idx.reshape(-1, k).long(), max(1, (1 << 27) // (k * Phi.shape[0]))):
        F = P[c]
        yield F @ F.transpose(1, 2)


def _extremes(e):
    lmin, lmax = e[:, 0], e[:, -1]
    return dict(lmin=lmin, lmax=lmax, delta=np.maximum(1 - lmin, lmax - 1), err=None)


def exact(case, seed):
    if sum(ns * k ** 3 for k, ns in _spans(case)) > 1.2e11 and case["path"] != "blocks":
        return None  # over a few seconds of LAPACK
    x = _inputs(case, seed)
    path, k = case["path"], case.get("k")
    if path == "blocks":
        return [torch.cat([b.cpu() for b in _gram_blocks(x["Phi"], x["idx"], k)]), None]
    if path == "gram":
        return _extremes(np.concatenate([_eigs(b) for b in _gram_blocks(x["Phi"], x["idx"], k)]))
    if path == "serve":
        mats = [_gram64(x["Phi"]).float(), _gram64(x["other"]).float()]
        return [_extremes(_submatrix_eigs(mats[i], idx, kk)) for i, kk, idx in x["reqs"]]
    A64 = _gram64(x["Phi"])
    if path == "dropin":
        e = _submatrix_eigs(A64, x["idx"], k)
        return dict(rc=None, eig=e.reshape(-1), det=e.prod(1))
    A = A64.float()
    if path == "csr":
        off = x["offsets"]
        ks = off[1:] - off[:-1]
        lmin = np.empty(case["nsets"])
        lmax = np.empty(case["nsets"])
        for kk in KVALUES:
            at = (ks == kk).nonzero().squeeze(1)
            if at.numel():
                S = x["idx"][off[:-1][at][:, None] + torch.arange(kk, device="cuda")]
                e = _submatrix_eigs(A, S, kk)
                lmin[at.cpu().numpy()], lmax[at.cpu().numpy()] = e[:, 0], e[:, -1]
        return dict(lmin=lmin, lmax=lmax, delta=np.maximum(1 - lmin, lmax - 1), err=None)
    e = _submatrix_eigs(A, x["idx"], k)
    out = _extremes(e)
    if path == "solve_all":
        out.update(eig=e.reshape(-1), det=e.prod(1))
    return out
