"""Epochs of the carry flags: a flag that an earlier run left in a batch's or a
service slot's flag array must not pass as this run's, so every run has an
epoch of its own (hg_epoch.h, compiled here) and every carry of a batch uses
its run's."""

import os
import re
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "hypergeometrica_gb300", "csrc")

PROGRAM = r"""
#include "hg_epoch.h"
#include <cstdio>
int main() {
  hg::ScanEpoch e;
  uint32_t before = 0;
  for (int i = 0; i < 100000; ++i) {
    const uint32_t k = e.next();
    if (k == 0 || k == hg::kPersistEpoch || k <= before) return 1;
    before = k;
  }
  e.last = 0xfffffffeu;  // around the end of the 32 bits
  if (e.next() != 0xffffffffu) return 2;
  const uint32_t k = e.next();
  if (k == 0 || k == hg::kPersistEpoch || k == 0xffffffffu) return 3;
  return 0;
}
"""


def test_epochs_differ_from_run_to_run(tmp_path):
    src = tmp_path / "epoch.cpp"
    src.write_text(PROGRAM)
    exe = str(tmp_path / "epoch")
    subprocess.run(["g++", "-std=c++17", "-I", CSRC, str(src), "-o", exe], check=True)
    assert subprocess.run([exe]).returncode == 0


def test_batches_and_slots_take_the_epoch_of_their_run():
    api = open(os.path.join(CSRC, "hg_api.cu")).read()
    svc = open(os.path.join(CSRC, "hg_service.cu")).read()
    run_group = api[api.index("int run_group("):api.index("BatchBufs batch_bufs(")]
    assert re.findall(r"ss\.epoch = (.*);", run_group) == ["bb.epoch"]
    made = re.findall(r"BatchBufs(?: bb)?\{[^}]*\}", api + svc)
    assert len(made) == 2 and all(m.rstrip("}").endswith("epoch.next()") for m in made), made
