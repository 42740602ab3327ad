"""The large-k kernels' exchange over many sets per cluster: its phases carry on
from set to set, whatever ends a set's steps early (an index outside the matrix
before the first step, a NaN in the submatrix in the middle of one, a
breakdown restart), so every other set must come out as it does alone, bit for
bit.  k at both ends of the 128 < k <= 192, 256 < k <= 384 and 384 < k <= 512
bins.
"""
import numpy as np
import pytest

from oracle import oracle as O
from paralanczos_b200 import _lib, api

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [129, 192, 257, 384, 385, 512])
def test_phases_across_sets(k):
    import torch
    n, nsets = 1200, 160  # more sets than clusters (or SMs) run at once
    rng = np.random.default_rng(k)
    Phi = rng.standard_normal((1024, n)) / np.sqrt(1024)
    A = (Phi.T @ Phi).astype(np.float32)
    A[n - 1, :] = np.nan  # sets with column n - 1 are not finite
    A[:, n - 1] = np.nan
    # columns n - 1 - k .. n - 2: an identity block, every step a breakdown
    lo = n - 1 - k
    A[lo:n - 1, :n - 1] = 0
    A[:n - 1, lo:n - 1] = 0
    A[np.arange(lo, n - 1), np.arange(lo, n - 1)] = 1
    _, idx = O.gen_stream(k, 0, nsets, lo, 0, k, k)
    idx = idx.reshape(nsets, k).copy()
    bad, nan, ident = range(0, nsets, 7), range(3, nsets, 11), range(5, nsets, 29)
    for s in nan:
        idx[s, k // 2] = n - 1
    for s in ident:
        idx[s] = np.arange(lo, n - 1)
    for s in bad:
        idx[s, k - 1] = n
    Ad = torch.from_numpy(A).cuda()
    got = api.solve(Ad, torch.from_numpy(idx.reshape(-1)).cuda(), k=k)
    got = {q: v.cpu().numpy() for q, v in got.items()}
    for s in range(nsets):
        want = (_lib.PL_SET_BAD_INDEX if s in bad else _lib.PL_SET_NONFINITE if s in nan else
                _lib.PL_SET_BREAKDOWN if s in ident else 0)
        # (beta may also fall below the breakdown threshold on an ordinary set
        # of large k; the status bit only reports the restart)
        bits = got["err"][s] if want == _lib.PL_SET_BREAKDOWN else got["err"][s] & ~_lib.PL_SET_BREAKDOWN
        assert bits == want, (s, got["err"][s], want)
        if want in (_lib.PL_SET_BAD_INDEX, _lib.PL_SET_NONFINITE):
            assert np.isnan(got["lmin"][s]) and np.isnan(got["lmax"][s])
    for s in (1, 2, 5, 6, 9, 100, 159):
        one = api.solve(Ad, torch.from_numpy(idx[s].copy()).cuda(), k=k)
        for q in ("lmin", "lmax", "delta", "err"):
            assert one[q].cpu().numpy()[0] == got[q][s], (s, q)
