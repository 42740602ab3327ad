"""The shipped kernel for 48 < k <= 64 reads ahead (the next set's triangle, staged
in shared memory behind this set's steps) and holds A_S in tensor memory.  Neither
changes an operation, so its results are bitwise those of the shape with the same
rows per thread and neither, in extremes and in all-eigenvalue mode, on a uniform
stream and on an uneven one with sets of an index outside [0, n) and of a k that is
another kernel's between prefetched neighbours.
"""
import numpy as np
import pytest

from oracle import oracle as O
from paralanczos_b200 import _lib, api

pytestmark = pytest.mark.gpu

KMAX = 64


def _variants():
    b = next(i for i in range(api.num_bins()) if api.bin_kmax(i) == KMAX)
    descs = [api.tune_describe(b, v)[1] for v in range(api.tune_describe(b, 0)[0])]
    shipped = next(v for v, d in enumerate(descs) if "prefetch tmem" in d)
    plain = next(v for v, d in enumerate(descs) if d.startswith("sharedA KB=64 RPT=2 CTA=128 MINB="))
    return b, shipped, plain


def _run(b, v, A, idx, every, **kw):
    import torch
    api.tune_set(b, v)
    try:
        out = api.solve(A, torch.from_numpy(idx).cuda(), want_all=every, **kw)
        torch.cuda.synchronize()
    finally:
        api.tune_set(b, -1)
    return {q: t.cpu().numpy() for q, t in out.items()}


def _matrix(seed):
    import torch
    rng = np.random.default_rng(seed)
    Phi = rng.standard_normal((512, 2048)) / np.sqrt(512)
    return torch.from_numpy((Phi.T @ Phi).astype(np.float32)).cuda()


def test_the_shipped_kernel_is_the_one_compared():
    b, shipped, _ = _variants()
    assert api.tune_get(b) == shipped


@pytest.mark.parametrize("every", [False, True])
@pytest.mark.parametrize("k", [49, 63, 64])
def test_uniform_bitwise(k, every):
    b, shipped, plain = _variants()
    A = _matrix(7)
    idx = O.gen_stream(31, 0, 6000, 2048, 0, k, k)[1]
    r, r0 = (_run(b, v, A, idx, every, k=k) for v in (shipped, plain))
    assert ((r["err"] & ~_lib.PL_SET_BREAKDOWN) == 0).all()
    for q in r:
        np.testing.assert_array_equal(r[q], r0[q], err_msg=q)


@pytest.mark.parametrize("every", [False, True])
def test_uneven_with_bad_sets_bitwise(every):
    import torch
    b, shipped, plain = _variants()
    A = _matrix(8)
    n, nsets = 2048, 5000
    rng = np.random.default_rng(9)
    parts, offs, bad = [], [0], []
    for s in range(nsets):
        k = 65 if s % 379 == 17 else int(rng.integers(49, 65))
        S = rng.choice(n, size=k, replace=False).astype(np.int32)
        if s % 211 == 5:
            S[k // 2] = n + 7 if s % 2 else -3
            bad.append(s)
        parts.append(S)
        offs.append(offs[-1] + k)
    idx, offsets = np.concatenate(parts), torch.tensor(offs).cuda()
    r, r0 = (_run(b, v, A, idx, every, offsets=offsets) for v in (shipped, plain))
    for s in bad:
        assert r["err"][s] == _lib.PL_SET_BAD_INDEX and np.isnan(r["lmin"][s])
    assert ((np.delete(r["err"], bad) & ~_lib.PL_SET_BREAKDOWN) == 0).all()
    for q in r:
        np.testing.assert_array_equal(r[q], r0[q], err_msg=q)  # (NaN equals NaN here)
