"""Gram blocks with several sets per 128-row tile (k <= 16, 32, 64, when there are
sets enough for every SM): the same bits as one set per tile (calls of few sets),
sets with an index outside the frame flagged on their own, a last tile that is
not full, and the solve on such blocks.
"""
import numpy as np
import pytest

from paralanczos_b200 import _lib, api

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [1, 8, 15, 16, 17, 31, 32, 33, 50, 63, 64, 65])
@pytest.mark.parametrize("m", [100, 640])
def test_packed_tiles_are_bitwise_single_tiles(k, m):
    import torch
    n, nsets = 900, 8 * 148 + 3
    rng = np.random.default_rng(7 * k + m)
    Phi = torch.from_numpy((rng.standard_normal((m, n)) / np.sqrt(m)).astype(np.float32)).cuda()
    idx = np.argsort(rng.random((nsets, n)), axis=1)[:, :k].astype(np.int32)
    bad = [0, 7, 8, 500, nsets - 1]
    idx[bad, k - 1] = [n, -1, n + 5, n, -3]
    f = api.GramFrame(Phi)
    B, err = f.blocks(torch.from_numpy(idx.reshape(-1)).cuda(), k)
    want = np.zeros(nsets, dtype=np.int32)
    want[bad] = _lib.PL_SET_BAD_INDEX
    np.testing.assert_array_equal(err.cpu().numpy(), want)
    B = B.cpu().numpy()
    for s0 in (0, 5, 600, nsets - 20):  # 20 sets: one per tile
        one, e1 = f.blocks(torch.from_numpy(np.ascontiguousarray(idx[s0:s0 + 20]).reshape(-1)).cuda(), k)
        ok = want[s0:s0 + 20] == 0
        np.testing.assert_array_equal(e1.cpu().numpy(), want[s0:s0 + 20])
        np.testing.assert_array_equal(one.cpu().numpy()[ok], B[s0:s0 + 20][ok])
    np.testing.assert_array_equal(B[want == 0], B[want == 0].transpose(0, 2, 1))
    out = f.solve(torch.from_numpy(idx.reshape(-1)).cuda(), k)
    np.testing.assert_array_equal(out["err"].cpu().numpy() & ~_lib.PL_SET_BREAKDOWN, want)
    e = np.linalg.eigvalsh(B[want == 0][:200].astype(np.float64))
    good = np.flatnonzero(want == 0)[:200]
    assert np.max(np.abs(out["lmin"].cpu().numpy()[good] - e[:, 0])) <= 1e-5 * np.max(e)
    assert np.max(np.abs(out["lmax"].cpu().numpy()[good] - e[:, -1])) <= 1e-5 * np.max(e)
