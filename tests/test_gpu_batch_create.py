"""Creating a batch sets up the schedule it will run, not both."""

import time

import numpy as np
import pytest

from hypergeometrica_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def test_default_batch_sets_up_one_schedule(hg):
    """A batch of four short products from creation to its end, as the one-shot
    call runs it.  The persistent schedule's set-up (a work list) is shorter
    than the per-pass one's (counts, flags, three streams and seven events), so
    a batch that runs persistently costs no more than one created per pass;
    with both set up it cost a fifth more."""
    import torch

    from hypergeometrica_gb300 import device as D

    items = []
    for k, n in enumerate((70, 200, 450, 1000)):
        x, y = (torch.from_numpy(W.limbs(70 + 2 * k + j, n).view(np.int64)).cuda() for j in range(2))
        items.append((x, y, torch.empty(2 * n, dtype=torch.int64, device="cuda")))

    def once(schedule):
        t0 = time.perf_counter()
        batch = D.Batch(items, autotune=False, schedule=schedule)
        batch.run()
        torch.cuda.synchronize()
        batch.close()
        return 1e6 * (time.perf_counter() - t0)

    outs = []
    for schedule in (None, "per_pass"):
        for _, _, out in items:
            out.fill_(-1)
        for _ in range(5):
            once(schedule)
        D.sync()
        outs.append([out.clone() for _, _, out in items])
    for a, b in zip(*outs):
        assert torch.equal(a, b)
    t = [(once(None), once("per_pass")) for _ in range(101)]
    default, per_pass = np.median(np.array(t), axis=0)
    assert default < per_pass, (default, per_pass)
