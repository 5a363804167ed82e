"""Runs of one batch, captured and not, in any order: each clears or tells apart
the carry flags that the runs before it left."""

import numpy as np
import pytest

from hypergeometrica_gb300 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("schedule", ["per_pass", "persistent"])
def test_replays_between_runs(hg, schedule):
    """Products of all-ones limbs, whose carries cross every tile, short and
    long carries (one launch and two) in one batch."""
    import torch

    from hypergeometrica_gb300 import device as D

    items = []
    for k, (nx, ny) in enumerate([(1500, 1400), (1 << 14, 3000), (1 << 18, 1 << 18), (300000, 200001)]):
        x, y = (torch.from_numpy(W.limbs(k, n, "ones").view(np.int64)).cuda() for n in (nx, ny))
        items.append((x, y, torch.empty(nx + ny, dtype=torch.int64, device="cuda")))
    want = []
    for x, y, out in items:
        D.mul(x, y, out)
        D.sync()
        want.append(out.clone())
    batch = D.Batch(items, autotune=False, schedule=schedule)
    stream = torch.cuda.Stream()
    batch.run(stream)
    stream.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        batch.run(stream)
    for step in ("replay", "replay", "run", "replay", "run", "run", "replay"):
        for _, _, out in items:
            out.fill_(-1)
        torch.cuda.synchronize()
        if step == "run":
            batch.run(stream)
        else:
            with torch.cuda.stream(stream):
                graph.replay()
        torch.cuda.synchronize()
        D.sync()
        for k, (_, _, out) in enumerate(items):
            assert torch.equal(out, want[k]), (step, k)
    batch.close()
