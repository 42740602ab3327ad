"""A set's eigenvalues do not depend on the call that it is in: calls of few and
of many sets, and calls with sets of other k, give the same bits.  Short calls
of 48 < k <= 64 in the all-eigenvalue mode run on another kernel than long ones;
the matrix is also one whose triangles differ in their last bits, of which
either kernel has to read the same one.
"""
import numpy as np
import pytest

from oracle import oracle as O
from paralanczos_b200 import api

pytestmark = pytest.mark.gpu

OUT = ("lmin", "lmax", "delta", "err", "eig", "det")


def _solve(At, idx, **kw):
    return {q: v.cpu().numpy() for q, v in api.solve(At, idx, want_all=True, **kw).items()}


@pytest.mark.parametrize("symmetric", [True, False])
@pytest.mark.parametrize("k", [16, 33, 49, 50, 57, 64, 65, 100])
def test_all_eigenvalues_alone_and_in_company(k, symmetric):
    import torch
    n, nsets = 500, 12_000
    rng = np.random.default_rng(40 + k)
    Phi = rng.standard_normal((300, n)) / np.sqrt(300)
    A = (Phi.T @ Phi).astype(np.float32)
    A[7:30, 7:30] = np.eye(23, dtype=np.float32)  # sets inside it break down
    A[7:30, 30:] = 0
    A[30:, 7:30] = 0
    A[7:30, :7] = 0
    A[:7, 7:30] = 0
    if not symmetric:
        A += np.triu(A, 1) * np.float32(2.0 ** -23)
    At = torch.from_numpy(A).cuda()
    idx = O.gen_stream(11, 0, nsets, n, 0, k, k)[1].reshape(nsets, k)
    it = torch.from_numpy(idx.reshape(-1).copy()).cuda()
    many = _solve(At, it, k=k)
    at = 0
    for m in (1, 2, 40, 300, 900, 2400):
        few = _solve(At, it[at * k:(at + m) * k].contiguous(), k=k)
        for q in OUT:
            w = k if q == "eig" else 1
            np.testing.assert_array_equal(few[q], many[q][at * w:(at + m) * w], err_msg=f"{q} of {m} sets")
        at += m
    # in a CSR call: 300 sets, others of k = 20 and 100 between them
    parts, offs = [], [0]
    for s in range(300):
        for S in (idx[s], rng.choice(n, 20, False), rng.choice(n, 100, False)):
            parts.append(np.asarray(S, np.int32))
            offs.append(offs[-1] + len(S))
    mix = _solve(At, torch.from_numpy(np.concatenate(parts)).cuda(), offsets=torch.tensor(offs).cuda())
    for q in OUT:
        if q == "eig":
            for s in range(300):
                np.testing.assert_array_equal(mix[q][offs[3 * s]:offs[3 * s] + k], many[q][s * k:(s + 1) * k])
        else:
            np.testing.assert_array_equal(mix[q][::3], many[q][:300], err_msg=q)
