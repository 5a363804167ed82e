"""hg_shutdown beside running sums: neither waits for a lock the other holds,
and a sum either completes with the right limbs or reports HG_ERR_NOT_INIT."""

import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

# 40 short sums (descriptors from the pool), two long ones (the library's scan
# state) and 50 lengths per call, from two threads on their own streams, while
# the main thread shuts the library down and starts it again.
PROGRAM = r"""
import ctypes, threading, time
import numpy as np, torch
import hypergeometrica_gb300 as H
from hypergeometrica_gb300._lib import HG_ERR_NOT_INIT, HgSum, HGError, check, load

H.init()
ones = torch.full((1 << 16,), -1, dtype=torch.int64, device="cuda")
one = torch.ones(1, dtype=torch.int64, device="cuda")
NS = [100] * 40 + [1 << 16] * 2
done, failures = [0, 0], []

def work(t):
    try:
        st = torch.cuda.Stream()
        outs = [torch.empty(n + 1, dtype=torch.int64, device="cuda") for n in NS]
        torch.cuda.synchronize()
        sums = (HgSum * len(NS))(*[HgSum(ones.data_ptr(), n, one.data_ptr(), 1, o.data_ptr(), n + 1, 1, 1)
                                  for n, o in zip(NS, outs)])
        vecs = np.array([[ones.data_ptr(), 1000 + k] for k in range(50)], dtype=np.uint64)
        res, sizes = np.empty((len(NS), 2), dtype=np.int64), np.empty(50, dtype=np.int64)
        while time.time() < end:
            res[:] = 0
            try:
                check(load().hg_sums_and_sizes(ctypes.addressof(sums), None, None, len(NS), res.ctypes.data,
                                               vecs.ctypes.data, 50, sizes.ctypes.data, st.cuda_stream))
            except HGError as e:
                if e.code != HG_ERR_NOT_INIT:
                    raise
                continue
            done[t] += 1
            assert (res[:, 1] == np.array(NS) + 1).all() and (res[:, 0] == 1).all(), res
            assert (sizes == 1000 + np.arange(50)).all()
    except BaseException as e:
        failures.append(e)

end = time.time() + 3
threads = [threading.Thread(target=work, args=(t,)) for t in range(2)]
for t in threads:
    t.start()
stops = 0
while time.time() < end:
    check(load().hg_shutdown())
    H.init()
    time.sleep(0.002)
    stops += 1
for t in threads:
    t.join()
assert not failures, failures
assert min(done) > 0 and stops > 3, (done, stops)
print("done", done, "shutdowns", stops)
"""


def test_sums_beside_shutdowns(hg):
    r = subprocess.run([sys.executable, "-c", PROGRAM], cwd=ROOT, capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
