"""CPU: the streams of a batch's single launches (grus_framework_gb300/csrc/
side_streams.h), compiled with g++: one stream per graph handle, whatever index
names it, and the handles in turn."""
import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parents[1]
DRIVER = r"""
#include <cstdio>
#include "side_streams.h"
int main() {
  int g[7];
  grus::SideStreams s(4);
  // graphs 0 and 1 are listed twice (by another index each)
  const int order[] = {0, 1, 0, 2, 1, 3, 4, 0, 5, 6, 4, 1};
  for (int i : order) std::printf("%d:%d ", i, s.of(&g[i]));
  std::printf("| %zu\n", s.graphs());
  return 0;
}
"""


def test_one_stream_per_handle(tmp_path):
    (tmp_path / "s.cpp").write_text(DRIVER)
    exe = tmp_path / "s"
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", str(ROOT / "grus_framework_gb300" / "csrc"),
                    str(tmp_path / "s.cpp"), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, check=True).stdout
    pairs, count = out.split("|")
    got = [tuple(map(int, p.split(":"))) for p in pairs.split()]
    streams = {}
    for graph, stream in got:
        assert streams.setdefault(graph, stream) == stream
    assert [streams[i] for i in range(7)] == [0, 1, 2, 3, 0, 1, 2]
    assert int(count) == 7


PLAN = r"""
#include <cstdio>
#include "side_streams.h"
int main() {
  int a[6];
  while (std::scanf("%d %d %d %d %d %d", a, a + 1, a + 2, a + 3, a + 4, a + 5) == 6) {
    const grus::SidePlan p = grus::plan_sides(a[0], a[1], a[2], a[3], a[4], a[5]);
    std::printf("%d %d %d\n", p.streams, p.workers, (int)p.beside);
  }
  return 0;
}
"""


def test_side_launches_fit_beside_the_workers(tmp_path):
    """Side launches of one CTA an SM and the workers' CTAs never need more slots
    than there are, whatever the order in which they start."""
    (tmp_path / "p.cpp").write_text(PLAN)
    exe = tmp_path / "p"
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", str(ROOT / "grus_framework_gb300" / "csrc"),
                    str(tmp_path / "p.cpp"), "-o", str(exe)], check=True)
    cases = [(4, per_sm, 152, cluster, per_sm * 152 // cluster, tasks)
             for per_sm in (0, 1, 2, 3, 4, 8) for cluster in (1, 3, 8, 16)
             for tasks in (0, 1, 5, 9, 10, 19, 20, 38, 39, 500)]
    out = subprocess.run([str(exe)], input="\n".join(" ".join(map(str, c)) for c in cases),
                         capture_output=True, text=True, check=True).stdout.splitlines()
    assert len(out) == len(cases)
    seen = set()
    for (most, per_sm, sms, cluster, workers, tasks), line in zip(cases, out):
        k, w, beside = map(int, line.split())
        assert 0 <= k <= min(most, per_sm)
        if beside:
            assert k >= 2 and 1 <= w <= workers and tasks <= 2 * w
            assert k * sms + w * cluster <= per_sm * sms
        else:
            assert w == workers
        seen.add((k, beside))
    assert {(4, 0), (3, 1), (2, 1)} <= seen
