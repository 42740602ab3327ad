"""The kernels that hold A[S,S] in tensor memory (k <= 64, 96, 128; the cluster
and symmetric-tile shapes are covered by test_cluster_shapes.py), each as its
bin's default: the values must be those of the general kernels, which read
A[S,S] from shared memory or registers.  k <= 64: the same FP32 sums, so the
same eigenvalues up to the FP64 sums of alpha and beta^2 (a few FP64 roundings:
1e-12 of the largest eigenvalue); k <= 128: another order of the FP32 row sums,
within 1e-5 of dsyev like every kernel.  Row, buffer and bin edges, invalid and
non-finite sets, breakdown restarts, leading dimension and pre-formed blocks.
"""
import numpy as np
import pytest

from oracle import oracle as O
from paralanczos_b200 import _lib, api

pytestmark = pytest.mark.gpu
RTOL = 1e-5


def _bin(k):
    return next(b for b in range(api.num_bins()) if k <= api.bin_kmax(b))


def _solve(A, idx, k, variant=None):
    import torch
    b = _bin(k)
    if variant is not None:
        api.tune_set(b, variant)
    try:
        out = api.solve(A, torch.from_numpy(np.ascontiguousarray(idx)).cuda(), k=k)
        torch.cuda.synchronize()
    finally:
        api.tune_set(b, -1)
    return {q: v.cpu().numpy() for q, v in out.items()}


@pytest.mark.parametrize("k", [49, 50, 63, 64, 65, 67, 95, 96, 97, 100, 127, 128])
def test_default_kernel_against_the_general_one(k):
    import torch
    n, nsets = 1500, 700
    rng = np.random.default_rng(k)
    Phi = rng.standard_normal((512, n)) / np.sqrt(512)
    A = (Phi.T @ Phi).astype(np.float32)
    A[n - 1, :] = np.nan
    A[:, n - 1] = np.nan
    lo = n - 1 - k  # an identity block: every step a breakdown
    A[lo:n - 1, :n - 1] = 0
    A[:n - 1, lo:n - 1] = 0
    A[np.arange(lo, n - 1), np.arange(lo, n - 1)] = 1
    _, idx = O.gen_stream(k, 0, nsets, lo, 0, k, k)
    idx = idx.reshape(nsets, k).copy()
    idx[::13, k - 1] = -1
    idx[3::17, 0] = n - 1
    idx[5::101] = np.arange(lo, n - 1)
    pad = torch.full((n, n + 3), float("nan"), device="cuda")
    pad[:, :n] = torch.from_numpy(A).cuda()
    At = pad[:, :n]
    got = _solve(At, idx.reshape(-1), k)
    ref = _solve(At, idx.reshape(-1), k, 0)
    np.testing.assert_array_equal(got["err"], ref["err"])
    bad = (got["err"] & ~_lib.PL_SET_BREAKDOWN) != 0
    assert bad.any() and not bad.all() and (got["err"] == _lib.PL_SET_BREAKDOWN).any()
    tol = 1e-12 if k <= 64 else RTOL
    for q in ("lmin", "lmax", "delta"):
        assert np.isnan(got[q][bad]).all()
        assert np.max(np.abs(got[q][~bad] - ref[q][~bad])) <= tol * np.max(ref["lmax"][~bad])
    ordinary = np.flatnonzero(got["err"] == 0)[:40]
    for s, t in zip(ordinary, O.dsyev_batch(A, idx[ordinary].reshape(-1), k=k)):
        assert abs(got["lmin"][s] - t[0]) <= RTOL * t[0] and abs(got["lmax"][s] - t[-1]) <= RTOL * t[-1]
    for s in ordinary[:3]:  # alone as among others
        one = _solve(At, idx[s], k)
        assert one["lmin"][0] == got["lmin"][s] and one["lmax"][0] == got["lmax"][s]


@pytest.mark.parametrize("k", [52, 64, 96, 112, 128])
def test_gram_blocks_in_tensor_memory(k):
    import torch
    rng = np.random.default_rng(k)
    Phi = torch.from_numpy((rng.standard_normal((300, 800)) / np.sqrt(300)).astype(np.float32)).cuda()
    _, idx = O.gen_stream(k, 0, 400, 800, 0, k, k)
    it = torch.from_numpy(idx).cuda()
    f = api.GramFrame(Phi)
    out = f.solve(it, k)
    B = f.blocks(it, k)[0].double()
    e = torch.linalg.eigvalsh(B).cpu().numpy()
    assert (out["err"].cpu().numpy() == 0).all()
    assert np.max(np.abs(out["lmin"].cpu().numpy() - e[:, 0]) / e[:, 0]) <= RTOL
    assert np.max(np.abs(out["lmax"].cpu().numpy() - e[:, -1]) / e[:, -1]) <= RTOL
