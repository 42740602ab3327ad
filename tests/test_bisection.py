"""Bisection of the tridiagonals: the extremes by one thread each (full queues)
or by several threads in tree rounds (queues of few sets, short calls), and the
all-eigenvalue mode (two eigenvalues per thread, blocks of 8 or 16 rows with
remainders).  The same sets in a large batch, in calls of 1, 2, 3 and 5 sets and
in the all-eigenvalue mode: every difference stays below 2^-33 of the
spectrum's scale, twice the bisection's tolerance (FP64 rounding moves an
interval's ends, never by more than its last width); eigenvalues against dsyev
within 1e-5 of the largest, and Det their product.
"""
import numpy as np
import pytest

from oracle import oracle as O
from paralanczos_b200 import _lib, api

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [1, 2, 3, 7, 8, 9, 15, 16, 17, 24, 31, 32, 33, 47, 48, 49, 63, 64, 65, 80, 96, 97,
                               127, 128])
def test_few_sets_and_all_eigenvalues_agree_with_the_batch(k):
    import torch
    n, nsets = 700, 5000
    rng = np.random.default_rng(1000 + k)
    Phi = rng.standard_normal((400, n)) / np.sqrt(400)
    A = (Phi.T @ Phi).astype(np.float32)
    _, idx = O.gen_stream(3 + k, 0, nsets, n, 0, k, k)
    At, it = torch.from_numpy(A).cuda(), torch.from_numpy(idx).cuda()
    batch = {q: v.cpu().numpy() for q, v in api.solve(At, it, k=k).items()}
    scale = 4.0 * np.max(batch["lmax"])  # at least the Gershgorin interval's ends
    tol = 2.0 ** -33 * scale
    assert ((batch["err"] & ~_lib.PL_SET_BREAKDOWN) == 0).all()
    at = 0
    for m in (1, 2, 3, 5):
        few = api.solve(At, it[at * k:(at + m) * k].contiguous(), k=k)
        for q in ("lmin", "lmax", "delta"):
            assert np.max(np.abs(few[q].cpu().numpy() - batch[q][at:at + m])) <= tol, (q, m)
        np.testing.assert_array_equal(few["err"].cpu().numpy(), batch["err"][at:at + m])
        at += m
    whole = {q: v.cpu().numpy() for q, v in api.solve(At, it, k=k, want_all=True).items()}
    eig = whole["eig"].reshape(nsets, k)
    assert (np.diff(eig, axis=1) >= 0).all()
    np.testing.assert_array_equal(eig[:, 0], whole["lmin"])
    np.testing.assert_array_equal(eig[:, -1], whole["lmax"])
    same_sums = k <= 64  # above, the all-eigenvalue kernels sum rows in another order
    lim = tol if same_sums else 1e-5 * scale
    assert np.max(np.abs(whole["lmin"] - batch["lmin"])) <= lim
    assert np.max(np.abs(whole["lmax"] - batch["lmax"])) <= lim
    np.testing.assert_allclose(whole["det"], np.prod(eig, axis=1), rtol=1e-12 * k)
    for s, t in enumerate(O.dsyev_batch(A, idx[:20 * k], k=k)):
        assert np.max(np.abs(eig[s] - t)) <= 1e-5 * t[-1]


@pytest.mark.parametrize("k", [1, 5, 6, 8, 9, 10, 11, 12, 13, 16, 18, 31, 33, 48, 50, 61, 64, 66, 95, 97, 126])
def test_rows_that_fill_up_a_tridiagonal_count_nothing(k):
    """T is filled up to a multiple of 4 rows above its spectrum.  A scaled by a
    power of two scales every step exactly, so the results scale within twice the
    bisection's tolerance; a zero matrix has the couplings of 2^-300 that its
    decoupled rows store, so eigenvalues of at most two of them (and the interval
    2^-51 wider).  Calls of few sets in
    all-eigenvalue mode (k = 49 .. 64: another kernel) agree with many."""
    import torch
    n, nsets = 300, 2000
    rng = np.random.default_rng(77 + k)
    Phi = rng.standard_normal((400, n)) / np.sqrt(400)
    At = torch.from_numpy((Phi.T @ Phi).astype(np.float32)).cuda()
    it = torch.from_numpy(O.gen_stream(5 + k, 0, nsets, n, 0, k, k)[1]).cuda()
    one = api.solve(At, it, k=k, want_all=True)
    scale = 4.0 * float(one["lmax"].max())
    for e in (-40, 40):
        f = 2.0 ** e
        for every in (False, True):
            got = api.solve(At * f, it, k=k, want_all=every)
            for q in ("lmin", "lmax"):
                lim = 2.0 ** -33 if every or k <= 64 else 1e-5
                assert float((got[q] / f - one[q]).abs().max()) <= lim * scale, (e, every, q)
            if every:
                assert float((got["eig"] / f - one["eig"]).abs().max()) <= 2.0 ** -33 * scale
    zero = api.solve(At * 0, it, k=k, want_all=True)
    assert float(zero["eig"].abs().max()) <= 2.0 ** -299 * (1 + 2.0 ** -50)
    for m in (1, 40, 1100):
        few = api.solve(At, it[:m * k].contiguous(), k=k, want_all=True)
        assert float((few["eig"] - one["eig"][:m * k]).abs().max()) <= 2.0 ** -33 * scale, m
