"""series.multiply hands addresses to the library, so it looks at its operands
first: limbs outside CUDA memory, strided limbs and a size past the tensor's
end must never reach a kernel.  On the CPU, against a stand-in for the library
that records the calls."""

import types

import pytest
import torch

from hypergeometrica_gb300 import series as S


class CudaTensor:
    """What multiply looks at in a CUDA tensor."""

    is_cuda = True

    def __init__(self, n, step=1):
        self.n, self.step = n, step

    def numel(self):
        return self.n

    def is_contiguous(self):
        return self.step == 1 or self.n <= 1

    def data_ptr(self):
        return 4096

    def __getitem__(self, s):
        return CudaTensor(min(self.n, s.stop), self.step)


@pytest.fixture
def calls(monkeypatch):
    made = []
    lib = types.SimpleNamespace(hg_mul_sized_device=lambda *a: made.append((a[1], a[3])) or 0)
    empty = torch.empty
    monkeypatch.setattr(S, "load", lambda: lib)
    monkeypatch.setattr(torch, "empty", lambda *a, device=None, **k: empty(*a, **k))
    monkeypatch.setattr(torch.cuda, "current_stream", lambda: types.SimpleNamespace(cuda_stream=0))
    return made


class Service:
    """A service that records what it is asked to multiply."""

    def __init__(self, made):
        self.made = made

    def mul(self, x, nx, y, ny, out, nout, st):
        self.made.append((nx, ny))
        return nout


@pytest.mark.parametrize("served", [False, True])
@pytest.mark.parametrize("bad", [torch.ones(300, dtype=torch.int64), CudaTensor(300, step=2)])
@pytest.mark.parametrize("place", ["x", "y", "square"])
def test_refused_operands(calls, served, bad, place):
    good, bad = S.DeviceInt(1, CudaTensor(300), 300), S.DeviceInt(1, bad, 300)
    x, y = {"x": (bad, good), "y": (good, bad), "square": (bad, bad)}[place]
    with pytest.raises(ValueError):
        S.multiply(x, y, Service(calls) if served else None)
    assert not calls


@pytest.mark.parametrize("served", [False, True])
def test_size_past_the_end_takes_what_is_there(calls, served):
    x, y = S.DeviceInt(1, CudaTensor(300), 400), S.DeviceInt(1, CudaTensor(250), 250)
    S.multiply(x, y, Service(calls) if served else None)
    assert calls == [(300, 250)]
