"""Calls on several streams, from one thread and from several, give what they give
one after the other: device-pointer calls return before their kernels run, and
the kernels' scratch (the bisection queues, the bins of uneven calls) is shared.
"""
import threading

import numpy as np
import pytest

from oracle import oracle as O
from paralanczos_b200 import api

pytestmark = pytest.mark.gpu


def _calls():
    """(A, idx, keywords) of calls that use the shared scratch, a millisecond or so each."""
    import torch
    n = 900
    rng = np.random.default_rng(3)
    Phi = rng.standard_normal((512, n)) / np.sqrt(512)
    At = torch.from_numpy((Phi.T @ Phi).astype(np.float32)).cuda()
    calls = []
    for i, (k, nsets) in enumerate([(8, 300_000), (12, 200_000), (30, 60_000), (64, 12_000), (40, 25_000),
                                    (100, 1_500), (64, 3), (16, 150_000)]):
        calls.append((At, torch.from_numpy(O.gen_stream(i, 0, nsets, n, 0, k, k)[1]).cuda(), dict(k=k)))
    offs, idx = O.gen_stream(77, 0, 20_000, n, 2, 4, 120)
    calls.insert(3, (At, torch.from_numpy(idx).cuda(), dict(offsets=torch.from_numpy(offs).cuda())))
    return calls


def _check(got, want):
    for g, w in zip(got, want):
        for q in w:
            np.testing.assert_array_equal(g[q].cpu().numpy(), w[q])


def test_streams_do_not_share_a_call_s_scratch():
    import torch
    calls = _calls()
    want = []
    for A, idx, kw in calls:
        want.append({q: v.cpu().numpy() for q, v in api.solve(A, idx, **kw).items()})
        torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in range(3)]
    for rnd in range(3):
        got = []
        for i, (A, idx, kw) in enumerate(calls):
            with torch.cuda.stream(streams[(i + rnd) % 3]):
                got.append(api.solve(A, idx, **kw))
        torch.cuda.synchronize()
        _check(got, want)

    def worker(w, res):
        with torch.cuda.stream(streams[w]):
            res[w] = [api.solve(A, idx, **kw) for A, idx, kw in calls[w:] + calls[:w]]

    res = {}
    ts = [threading.Thread(target=worker, args=(w, res)) for w in range(3)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    torch.cuda.synchronize()
    for w in range(3):
        _check(res[w], want[w:] + want[:w])
