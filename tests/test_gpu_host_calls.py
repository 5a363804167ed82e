"""Host-memory products cost about what their device work and their copies do,
at every length and for page-locked and pageable buffers alike."""

import ctypes
import time

import numpy as np
import pytest

from hypergeometrica_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def _median_us(call, n):
    for _ in range(3):
        call()
    t = []
    for _ in range(n):
        t0 = time.perf_counter()
        call()
        t.append(time.perf_counter() - t0)
    return 1e6 * float(np.median(t))


def test_quadratic_product_reads_device_memory(hg, oracle):
    """16000 x 16000 limbs by the quadratic method take about 9 ms of kernel
    time on device operands; read over the host link, three times that.  The
    copies are 0.5 MB, below 100 us."""
    import torch

    from hypergeometrica_gb300 import device as D
    from hypergeometrica_gb300._lib import check, load

    n = 16000
    x, y = W.limbs(1, n), W.limbs(2, n)
    out = np.full(2 * n, 7, dtype=np.uint64)
    dx, dy = (torch.from_numpy(a.view(np.int64)).cuda() for a in (x, y))
    dout = torch.empty(2 * n, dtype=torch.int64, device="cuda")

    def host():
        check(load().hg_mul_schoolboy(x.ctypes.data, n, y.ctypes.data, n, out.ctypes.data, 2 * n))

    def device():
        D.mul_schoolboy(dx, dy, dout)
        D.sync()

    th, td = _median_us(host, 9), _median_us(device, 9)
    assert np.array_equal(out, dout.cpu().numpy().view(np.uint64))
    assert np.array_equal(out, oracle.mpz_mul_ntt(x, y)[:2 * n])
    assert th < 1.25 * td + 100, (th, td)


@pytest.mark.parametrize("pinned", [False, True])
@pytest.mark.parametrize("n", [4095, 4096, 32767, 32768, 131000])
def test_by_digit_at_the_ends_of_the_staged_sizes(hg, pinned, n):
    """A product by a digit moves 16 n bytes over a link of about 200 GB/s beside
    what the shortest one costs (25 us): twice that, and the driver's copies of
    pageable memory, hold it below 2 x + 40 us.  Copied on the host both ways,
    131000 limbs take 150 us."""
    import torch

    from hypergeometrica_gb300._lib import check, load

    d = 12345678901234567

    def buffers(k):
        x, out = W.limbs(3, k), np.full(k + 1, 7, dtype=np.uint64)
        if pinned:
            x, out = (torch.from_numpy(a.view(np.int64)).pin_memory().numpy().view(np.uint64) for a in (x, out))
        return x, out

    def call(x, out):
        return lambda: check(load().hg_mul_digit(x.ctypes.data, len(x), ctypes.c_uint64(d), out.ctypes.data, len(out)))

    x0, out0 = buffers(256)
    x, out = buffers(n)
    t0, t = _median_us(call(x0, out0), 31), _median_us(call(x, out), 31)
    want = int.from_bytes(x.tobytes(), "little") * d
    assert int.from_bytes(out.tobytes(), "little") == want
    assert t < 2 * t0 + 40, (t, t0)
