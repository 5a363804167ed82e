"""A product that a client only polls (hg_svc_status) is retired on time also
when another client has just left a wait: the worker looks at its batches at
least every 20 microseconds when no waiting client does."""

import time

import numpy as np
import pytest

from hypergeometrica_gb300 import workloads as W

pytestmark = pytest.mark.gpu

ROUNDS = 60
# The worker sleeps 20 us between looks; the rest is for the wake-up of its
# thread.  Asleep for 500 us, it would be 200 us late at the median.
LATE_US = 100.0


def test_polled_product_after_a_wait(hg):
    import torch

    from hypergeometrica_gb300 import device as D

    def square(n, seed):
        x = torch.from_numpy(W.limbs(seed, n).view(np.int64)).cuda()
        return x, None, torch.empty(2 * n, dtype=torch.int64, device="cuda")

    polled, waited = square(1 << 20, 1), square(200, 2)
    torch.cuda.synchronize()

    def seen(svc, wait):
        """Microseconds from the submission of `polled` until its status changes."""
        t0 = time.perf_counter()
        (a,) = svc.submit([polled])
        while svc.stats()["pending"]:  # admitted: it has a slot of its own
            pass
        (b,) = svc.submit([waited])
        if wait:
            svc.wait(b)
        while svc.status(a) == 0:
            pass
        t = 1e6 * (time.perf_counter() - t0)
        svc.wait_all()
        return t

    with D.Service(workspace_bytes=512 << 20, slots=2) as svc:
        for wait in (False, True):
            for _ in range(5):
                seen(svc, wait)
        alone, after = [], []
        for _ in range(ROUNDS):
            alone.append(seen(svc, False))
            after.append(seen(svc, True))
    assert np.median(after) < np.median(alone) + LATE_US, (np.median(after), np.median(alone))
