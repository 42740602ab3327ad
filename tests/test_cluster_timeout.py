"""The exchange between the CTAs of a set (k > 128) gives up after 2 s.  With one
CTA of every cluster held back from the steps (a test switch) its peers' waits
run out; with one that gives up behind a set's last step, its peers have all
they need and learn of it at the barrier.  Either way the cluster's CTAs leave
together: every set comes back as timed out (NaN and the status bit), sets of a
k out of range keep their own bit, the host-buffer call reports it, and the
next call in the same process solves everything.  Sets that time out after a
first breakdown are among them (the identity block's).
"""
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
pytestmark = pytest.mark.gpu

_SCRIPT = r"""
import os, sys
import numpy as np, torch
sys.path.insert(0, {root!r})
from oracle import oracle as O
from paralanczos_b200 import _lib, api
k, hold = {k}, {hold!r}
n, nsets = 700, 130                       # more sets than clusters run at once
rng = np.random.default_rng(k)
Phi = rng.standard_normal((1024, n)) / 32.0
A = (Phi.T @ Phi).astype(np.float32)
A[:k, :] = 0
A[:, :k] = 0
A[np.arange(k), np.arange(k)] = 1.0       # every step of set 1 breaks down
_, idx = O.gen_stream(k, 0, nsets, n, 0, k, k)
idx = idx.reshape(nsets, k).copy()
idx[1] = np.arange(k)
At, it = torch.from_numpy(A).cuda(), torch.from_numpy(idx.reshape(-1)).cuda()
good = {{q: v.cpu().numpy() for q, v in api.solve(At, it, k=k).items()}}
assert ((good["err"] & ~_lib.PL_SET_BREAKDOWN) == 0).all()
os.environ["PL_CLUSTER_TEST_HOLD"] = hold
lost = {{q: torch.full((nsets,), 7, dtype=torch.int32 if q == "err" else torch.float64, device="cuda")
        for q in ("lmin", "lmax", "delta", "err")}}
api.solve(At, it, k=k, out=lost)
torch.cuda.synchronize()
assert (lost["err"] == _lib.PL_SET_TIMEDOUT).all(), lost["err"]
for q in ("lmin", "lmax", "delta"):
    assert torch.isnan(lost[q]).all(), q
try:
    api.solve_host(A, idx.reshape(-1), k=k)
    sys.exit("no timeout reported")
except _lib.PLError as e:
    assert e.status == _lib.PL_ETIMEDOUT, e.status
os.environ["PL_CLUSTER_TEST_HOLD"] = "0"
again = api.solve(At, it, k=k)
host = api.solve_host(A, idx.reshape(-1), k=k)
for q in good:
    np.testing.assert_array_equal(again[q].cpu().numpy(), good[q])
    np.testing.assert_array_equal(host[q], good[q])
print("ok")
"""


@pytest.mark.parametrize("k", [300, 480])
@pytest.mark.parametrize("hold", ["1", "2"])
def test_lost_clusters_report_every_set(k, hold):
    r = subprocess.run([sys.executable, "-c", _SCRIPT.format(root=ROOT, k=k, hold=hold)], capture_output=True,
                       text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip().endswith("ok"), r.stdout + r.stderr
