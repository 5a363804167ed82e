"""A batch whose groups do not fit the free device memory together runs them
one after another, on the workspace of its largest group."""

import numpy as np
import pytest

from hypergeometrica_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def test_batch_falls_back_to_one_group_at_a_time(hg):
    """Pairs and squares of 2^20 to 2^23 limbs are eight groups of which the
    largest takes a third of the memory of all.  A first batch with room
    builds the tables and gives the expected limbs."""
    import torch

    from hypergeometrica_gb300 import device as D

    items = []
    for k, bits in enumerate((20, 21, 22, 23)):
        x, y = (torch.from_numpy(W.limbs(90 + 2 * k + j, 1 << bits).view(np.int64)).cuda() for j in range(2))
        items += [(x, y, torch.empty(2 << bits, dtype=torch.int64, device="cuda")),
                  (x, None, torch.empty(2 << bits, dtype=torch.int64, device="cuda"))]
    D.mul(items[6][0], items[6][1], items[6][2])
    D.sync()
    single = items[6][2].clone()
    room = torch.cuda.mem_get_info()[0]
    batch = D.Batch(items, autotune=False, schedule="per_pass")
    held = room - torch.cuda.mem_get_info()[0]  # all groups' workspace, descriptors and flags
    batch.run()
    D.sync()
    batch.close()
    want = [out.clone() for _, _, out in items]
    assert torch.equal(want[6], single)
    for _, _, out in items:
        out.fill_(-1)
    free = torch.cuda.mem_get_info()[0]
    filler = torch.empty(free - held * 2 // 3, dtype=torch.uint8, device="cuda")
    try:
        batch = D.Batch(items, autotune=False, schedule="per_pass")
        batch.run()
        D.sync()
        batch.close()
    finally:
        del filler
        torch.cuda.empty_cache()
    for k, (_, _, out) in enumerate(items):
        assert torch.equal(out, want[k]), k
