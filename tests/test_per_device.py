"""CPU: values found out once per device (grus_framework_gb300/csrc/per_device.h),
compiled with g++.  What is set on one device must be set again on the next, from
whichever thread its first call comes."""
import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parents[1]
DRIVER = r"""
#include <atomic>
#include <cstdio>
#include <thread>
#include <vector>
#include "per_device.h"
int main() {
  grus::PerDevice<int> p;
  std::atomic<int> finds[3] = {};
  auto get = [&](int dev) {
    int v = -1;
    const int rc = p.get(dev, &v, [&](int &x) {
      ++finds[dev];
      x = 10 + dev;
      return 0;
    });
    return rc ? -2 : v;
  };
  std::vector<std::thread> t;
  for (int i = 0; i < 12; ++i)
    t.emplace_back([&, i] {
      for (int k = 0; k < 100; ++k)
        if (get((i + k) % 3) != 10 + (i + k) % 3) std::puts("wrong value");
    });
  for (auto &x : t) x.join();
  for (int d = 0; d < 3; ++d)
    if (finds[d] != 1) std::printf("device %d found out %d times\n", d, finds[d].load());
  // a failure is reported and tried again; no device: nothing is kept
  int v = 0, tries = 0;
  auto failing = [&](int &x) { x = 7; return ++tries < 3 ? -1 : 0; };
  if (p.get(5, &v, failing) != -1 || p.get(5, &v, failing) != -1) std::puts("failure lost");
  if (p.get(5, &v, failing) != 0 || v != 7 || p.get(5, &v, failing) != 0 || tries != 3) std::puts("retry");
  if (p.get(-1, &v, failing) != 0 || p.get(-1, &v, failing) != 0 || tries != 5) std::puts("no device");
  return 0;
}
"""


def test_found_out_once_per_device(tmp_path):
    (tmp_path / "d.cpp").write_text(DRIVER)
    exe = tmp_path / "d"
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-I",
                    str(ROOT / "grus_framework_gb300" / "csrc"), str(tmp_path / "d.cpp"), "-o", str(exe)],
                   check=True)
    assert subprocess.run([str(exe)], capture_output=True, text=True, check=True).stdout == ""


def test_kernel_attributes_are_set_per_device():
    """Every place that sets a kernel's attributes does so through PerDevice (or
    in a function that only such a place calls)."""
    src = ROOT / "grus_framework_gb300" / "csrc"
    setters = {p.name: p.read_text().count("cudaFuncSetAttribute(") for p in src.glob("*.cu*")}
    setters = {k: v for k, v in setters.items() if v}
    assert setters == {"batch.cu": 1, "narrow.cuh": 2, "pagerank.cu": 1}
    for name in ("batch.cu", "pagerank.cu"):
        text = (src / name).read_text()
        at = text.index("cudaFuncSetAttribute(")
        assert ".get(current_device()" in text[at - 400:at]
    calls = [line for p in src.glob("*.cu") for line in p.read_text().splitlines()
             if "cluster_size(" in line and "narrow::" in line]
    assert calls and all(line.strip().startswith("v = ") for line in calls)
