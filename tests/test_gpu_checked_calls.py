"""Calls that wait for the device report what the checked build's kernels found
(libhg_gb300_checked.so), as hg_sync does: the range fault of a spectrum input
above its prime must not wait for some later call."""

import os
import subprocess
import sys

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

SCRIPT = r"""
import numpy as np
import torch

import hypergeometrica_gb300 as H
from hypergeometrica_gb300 import _lib, mpd, series
from hypergeometrica_gb300 import device as D
from hypergeometrica_gb300 import workloads as W

assert _lib.load().hg_build_checked() == 1, "the regular build was loaded"
H.init(0)
a, b = series.DeviceInt.from_int(3 << 20000), series.DeviceInt.from_int(5 << 9000)
for call in (lambda: series.multiply(a, b), lambda: mpd.mpz_add(a, b)):
    v = W.splitmix64(5, 1 << 13) >> np.uint64(2)
    v[17] = np.uint64(2 ** 64 - 1)  # above every prime
    t = torch.from_numpy(v.view(np.int64)).cuda()
    D.ntt_forward(t, 0)
    try:
        call()
        raise SystemExit("an input >= p went unreported")
    except _lib.HGError as e:
        assert e.code == _lib.HG_ERR_INCONSISTENT and "range" in str(e), e
    D.sync()  # the report cleared the fault words
assert series.multiply(a, b).to_int() == 15 << 29000
assert mpd.mpz_add(a, b).to_int() == (3 << 20000) + (5 << 9000)
print("reported")
"""


def test_waiting_calls_report_checked_faults(hg):
    from hypergeometrica_gb300 import build as B

    B.build(checked=True)
    r = subprocess.run([sys.executable, "-c", SCRIPT], env=dict(os.environ, HG_CHECKED="1", PYTHONPATH=ROOT),
                       capture_output=True, text=True, timeout=600)
    assert r.returncode == 0 and "reported" in r.stdout, r.stdout[-3000:] + r.stderr[-3000:]
