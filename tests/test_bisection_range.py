"""Counts of eigenvalues on matrices far from unit scale.  A scaled by 2^e scales
T by 2^e, and the minors of T - xI by 2^e a row, so a count that goes on for too
many rows without a rescaling over- or underflows.  Sizes with 0 to 3 rows
behind the last block of the counts, in every bin above 128 and some below; the
FP32 recurrence holds at these scales (beta^2 and products of two elements stay
in its range, down to subnormal ones that are 2^-31 of a sum), so the scaled
results agree within the FP32 recurrence's 1e-5.  The symmetric-tile engine,
192 < k <= 256, forms w^T A w of an unnormalised w in FP32 and holds to 2^+-40.
"""
import numpy as np
import pytest

from oracle import oracle as O
from paralanczos_b200 import _lib, api

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k,e", [(k, e) for k in (14, 30, 35, 50, 67, 99, 126, 129, 130, 131, 147, 163, 192, 259,
                                                  291, 387, 403, 507) for e in (-58, -54, 54)] +
                         [(k, e) for k in (193, 195, 211, 256) for e in (-36, 36)])
def test_extremes_scale_with_the_matrix(k, e):
    import torch
    n, nsets, m = 900, 40, 2 * k + 64
    rng = np.random.default_rng(500 + k)
    Phi = rng.standard_normal((m, n)) / np.sqrt(m)
    At = torch.from_numpy((Phi.T @ Phi).astype(np.float32)).cuda()
    it = torch.from_numpy(O.gen_stream(9 + k, 0, nsets, n, 0, k, k)[1]).cuda()
    one = api.solve(At, it, k=k)
    got = api.solve(At * 2.0 ** e, it, k=k)
    assert int((got["err"] & ~_lib.PL_SET_BREAKDOWN).abs().max()) == 0
    for q in ("lmin", "lmax"):
        assert float((got[q] * 2.0 ** -e - one[q]).abs().max()) <= 1e-5 * float(one["lmax"].max()), q
    truth = O.dsyev_batch(At.cpu().numpy(), it.cpu().numpy()[:3 * k], k=k)
    for s, t in enumerate(truth):
        assert abs(float(got["lmin"][s]) * 2.0 ** -e - t[0]) <= 1e-5 * t[-1]
        assert abs(float(got["lmax"][s]) * 2.0 ** -e - t[-1]) <= 1e-5 * t[-1]
