"""A kernel's shared memory limit and its resident CTAs belong to a device: a process with contexts on
several devices finds them on each (the bookkeeping, in a host program with stand-in devices and
threads), and no launcher keeps them in a plain static."""
from __future__ import annotations

import os
import re
import subprocess

from tests.conftest import ROOT

CSRC = os.path.join(ROOT, "camille_b200", "csrc")

PROGRAM = r"""
#include <cstdio>
#include <thread>
#include <vector>
#include "lee_per_device.h"
int main() {
  lee::PerDevice p;
  std::atomic<int> calls[70] = {};
  auto of = [&](int d) { return p.get(d, [&] { ++calls[d]; return 100 + d; }); };
  // one device after another, as contexts on both would launch
  for (int turn = 0; turn < 3; ++turn)
    for (int d : {0, 1, 7, 63})
      if (of(d) != 100 + d) return 1;
  for (int d : {0, 1, 7, 63})
    if (calls[d] != 1) return 2;
  // beyond the table: found again at every launch
  if (of(66) != 166 || of(66) != 166 || calls[66] != 2) return 3;
  // a failure is no answer
  lee::PerDevice q;
  if (q.get(2, [] { return 0; }) != 0 || q.get(2, [] { return 5; }) != 5 || q.get(2, [] { return 9; }) != 5) return 4;
  // threads that drive different devices
  lee::PerDevice r;
  std::atomic<int> bad{0};
  std::vector<std::thread> t;
  for (int w = 0; w < 8; ++w)
    t.emplace_back([&, w] {
      for (int k = 0; k < 20000; ++k)
        if (r.get((w + k) % 5, [&] { return 1 + (w + k) % 5; }) != 1 + (w + k) % 5) ++bad;
    });
  for (auto& x : t) x.join();
  if (bad) return 5;
  puts("ok");
  return 0;
}
"""


def test_the_bookkeeping_per_device(tmp_path):
    src, exe = tmp_path / "p.cpp", tmp_path / "p"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.returncode


def test_no_launcher_keeps_a_devices_facts_in_a_plain_static():
    for name in sorted(os.listdir(CSRC)):
        if name.endswith((".cu", ".cuh")):
            text = open(os.path.join(CSRC, name)).read()
            assert not re.search(r"^\s+static (bool|int|size_t)\b[^(]*;", text, re.M), name
