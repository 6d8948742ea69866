"""The first sorts of a process from several host threads at once, each on its own stream."""
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHILD = r"""
import ctypes, threading
import numpy as np, torch
from thrustrtc_b200 import _native as N
torch.cuda.init()
n, go, bad = 592 * 5120 + 77, threading.Barrier(12), []
def work(i):
    rng = np.random.default_rng(i)
    k = rng.integers(0, 1 << 31, n).astype(np.uint32 if i % 2 else np.int64)
    s = torch.cuda.Stream()
    with torch.cuda.stream(s):
        tk = torch.from_numpy(k.view(np.int32 if i % 2 else np.int64)).cuda()
        tv = torch.arange(n, dtype=torch.int32, device="cuda")
    s.synchronize()
    order = np.argsort(k, kind="stable")
    go.wait()
    p = lambda t: ctypes.c_void_p(t.data_ptr())
    st = ctypes.c_void_p(s.cuda_stream)
    ok = N.lib.trtc_raw_sort_by_key(5 if i % 2 else 6, p(tk), p(tv), 4, n, 0, st) == 0 and N.lib.trtc_raw_sync(st) == 0
    if not ok or tk.cpu().numpy().tobytes() != k[order].tobytes() or not (tv.cpu().numpy() == order).all():
        bad.append(i)
ts = [threading.Thread(target=work, args=(i,)) for i in range(12)]
[t.start() for t in ts]
[t.join() for t in ts]
assert not bad, bad
"""


@pytest.mark.gpu
def test_first_sorts_from_many_threads(cuda):
    r = subprocess.run([sys.executable, "-c", CHILD], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
