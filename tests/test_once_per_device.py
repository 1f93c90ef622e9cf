"""Kernel attributes are per device: the guard around their setters (gpview_gb300/csrc/gpv_once.h) runs
once for each device of a process, again after a failure, and holds every thread until it has run.  The
devices and the setter are made up, so this needs no GPU."""
import os
import re
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "gpview_gb300", "csrc")

PROGRAM = r"""
#include <cstdio>
#include <thread>
#include <vector>
#include "gpv_once.h"
int main() {
  gpv::OncePerDevice once;
  int calls[100] = {};
  bool ok[100] = {};  // the fake devices' attribute
  auto launch = [&](int dev, bool works) {
    once(dev, [&] { ++calls[dev]; ok[dev] = works; return works; });
    return ok[dev];
  };
  for (int r = 0; r < 3; ++r)
    for (int dev = 0; dev < 4; ++dev)
      if (!launch(dev, true)) return 1;
  for (int dev = 0; dev < 4; ++dev)
    if (calls[dev] != 1) return 2;
  if (launch(9, false) || !launch(9, true) || calls[9] != 2) return 3;   // a refusal is not remembered
  if (!launch(70, true) || !launch(70, true)) return 4;                  // past the flags: every time
  // threads that come at once: none goes on before its device's setter has run
  gpv::OncePerDevice shared;
  std::atomic<int> set[8], bad{0};
  for (auto &s : set) s = 0;
  std::vector<std::thread> th;
  for (int t = 0; t < 32; ++t)
    th.emplace_back([&, t] {
      const int dev = t % 8;
      shared(dev, [&] { set[dev].fetch_add(1); return true; });
      if (set[dev].load() == 0) bad.fetch_add(1);
    });
  for (auto &x : th) x.join();
  std::puts(bad.load() == 0 ? "ok" : "bad");
  return bad.load() ? 5 : 0;
}
"""


def test_once_for_each_device(tmp_path):
    src, exe = tmp_path / "once.cpp", tmp_path / "once"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and r.stdout.strip() == "ok", (r.returncode, r.stdout)


def test_attributes_are_set_through_it():
    for name in sorted(os.listdir(CSRC)):
        text = open(os.path.join(CSRC, name)).read()
        calls = len(re.findall(r"cudaFuncSetAttribute\(", text))
        assert calls == (1 if name == "gpv_internal.h" else 0), name
