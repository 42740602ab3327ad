"""Breakdown restarts of the large-k kernels: sets of columns whose frame rows have
rank 0.9 k break down late, and again in nearly every step from there on.  The
clusters restart from P's diagonal and one of its rows, formed anew from the steps'
vectors (one CTA per set: from P itself).  Such sets among ordinary ones, at both
ends of each bin: extremes against dsyev within 1e-5 of the largest, the same bits
alone and in company, the status bit on them.
"""
import numpy as np
import pytest

from oracle import oracle as O
from paralanczos_b200 import _lib, api

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [129, 150, 192, 257, 300, 384, 385, 450, 512])
def test_late_breakdowns(k):
    import torch
    n, nsets = 1400, 100
    rng = np.random.default_rng(k)
    Phi = rng.standard_normal((1024, n)) / 32.0
    Phi[int(0.9 * k):, n // 2:] = 0.0
    A = (Phi.T @ Phi).astype(np.float32)
    low = np.arange(nsets) % 3 == 1
    idx = np.stack([rng.choice(n // 2, k, replace=False) + (n // 2 if low[s] else 0)
                    for s in range(nsets)]).astype(np.int32)
    At = torch.from_numpy(A).cuda()
    got = {q: v.cpu().numpy() for q, v in api.solve(At, torch.from_numpy(idx.reshape(-1)).cuda(), k=k).items()}
    assert ((got["err"] & ~_lib.PL_SET_BREAKDOWN) == 0).all()
    assert (got["err"][low] == _lib.PL_SET_BREAKDOWN).all()
    sample = [0, 1, 4, 5, 97]
    for s, t in zip(sample, O.dsyev_batch(A, idx[sample].reshape(-1), k=k)):
        assert abs(got["lmin"][s] - t[0]) <= 1e-5 * t[-1], s
        assert abs(got["lmax"][s] - t[-1]) <= 1e-5 * t[-1], s
    for s in (1, 2, 49, 97):
        one = api.solve(At, torch.from_numpy(idx[s].copy()).cuda(), k=k)
        for q in got:
            assert one[q].cpu().numpy()[0] == got[q][s], (s, q)
