"""Many clients of one service: waiting clients leave its work to the worker, whose
batches then gather the products that arrive meanwhile."""

import threading

import numpy as np
import pytest

from hypergeometrica_gb300 import workloads as W

pytestmark = pytest.mark.gpu

CLIENTS, ROUNDS, LIMBS = 16, 150, 4000


def test_many_clients_share_batches(hg):
    """Sixteen threads that each submit one product and wait for it.  With every
    client enqueuing its own product a batch holds 1.15 of them, with the worker
    alone 1.6; a fifth of the products per second go with the difference."""
    import torch

    from hypergeometrica_gb300 import device as D

    items, want = [], []
    for k in range(CLIENTS):
        x, y = (torch.from_numpy(W.limbs(40 + 2 * k + j, LIMBS).view(np.int64)).cuda() for j in range(2))
        items.append((x, y, torch.full((2 * LIMBS,), -1, dtype=torch.int64, device="cuda")))
        want.append(torch.empty(2 * LIMBS, dtype=torch.int64, device="cuda"))
        D.mul(x, y, want[k])
    D.sync()
    torch.cuda.synchronize()
    failures = []
    with D.Service(workspace_bytes=1 << 30, slots=2) as svc:
        def client(k):
            try:
                for _ in range(ROUNDS):
                    (t,) = svc.submit([items[k]])
                    svc.wait(t)
            except BaseException as e:
                failures.append(e)

        threads = [threading.Thread(target=client, args=(k,)) for k in range(CLIENTS)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        st = svc.stats()
    assert not failures, failures
    assert st["completed"] == CLIENTS * ROUNDS and st["failed"] == 0
    for k, (_, _, out) in enumerate(items):
        assert torch.equal(out, want[k]), k
    assert st["completed"] > 1.3 * st["batches"], (st["completed"], st["batches"])
