"""Services opened as tight as their products allow (hg_svc_open): what
hg_svc_submit accepts must run, whatever tiles the carries of the batch take."""

import numpy as np
import pytest

from hypergeometrica_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def _squares(sizes):
    import torch

    items = []
    for k, n in enumerate(sizes):
        x = torch.from_numpy(W.limbs(500 + k, n).view(np.int64)).cuda()
        items.append((x, None, torch.full((2 * n,), -1, dtype=torch.int64, device="cuda")))
    torch.cuda.synchronize()
    return items


# A square of N points admits with 3 N words and its carry takes N / 1024 flag
# words up to 2^18 points: 14 and 13 sixteenths of 2^18 points (224 and 208
# words), and four lengths at once, each at the 256 tiles of a short carry.
@pytest.mark.parametrize("workspace, slots, max_batch, sizes", [
    (3 * 8 << 18, 1, 1, [114652]),
    (3 * 8 << 18, 1, 4, [1 << 17]),
    (64 << 20, 2, 64, [32768] * 4 + [16384] * 8 + [8192] * 16 + [4096] * 32),
])
def test_squares_in_a_tight_slot(hg, workspace, slots, max_batch, sizes):
    import torch

    from hypergeometrica_gb300 import device as D

    items = _squares(sizes)
    with D.Service(workspace_bytes=workspace, slots=slots, max_batch=max_batch) as svc:
        tickets = svc.submit(items)
        for t in tickets:
            svc.wait(t, timeout=60)
    for k, (x, _, out) in enumerate(items):
        want = torch.empty_like(out)
        D.sqr(x, want)
        D.sync()
        assert torch.equal(out, want), k
