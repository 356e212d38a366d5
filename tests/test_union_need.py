"""CPU: the workspace that a batch makes for its packs at creation
(union_need, grus_framework_gb300/csrc/union_plan.h, compiled with g++) holds
whatever launches plan_union makes of any queries on its graphs."""
import subprocess
from pathlib import Path

import numpy as np
import pytest

ROOT = Path(__file__).resolve().parents[1]
DRIVER = r"""
#include <cstdio>
#include "union_plan.h"
using namespace grus;
int main() {
  size_t G, Q;
  unsigned long long cap, maxg;
  while (scanf("%zu %zu %llu %llu", &G, &Q, &cap, &maxg) == 4) {
    std::vector<uint64_t> gn(G), gm(G);
    std::vector<bool> alone(G);
    for (size_t g = 0; g < G; ++g) {
      unsigned long long n, m;
      int a;
      if (scanf("%llu %llu %d", &n, &m, &a) != 3) return 2;
      gn[g] = n, gm[g] = m, alone[g] = a;
    }
    const UnionNeed need = union_need(gn, gm, alone, cap);
    std::vector<int> q(Q);
    std::vector<uint32_t> qg(Q);
    for (size_t i = 0; i < Q; ++i) {
      q[i] = (int)i;
      if (scanf("%u", &qg[i]) != 1) return 2;
    }
    const UnionPlan p = plan_union(q, qg, gn, gm, cap, maxg, 128);
    for (const auto &l : p.launches) {
      if (l.size() == 1 && !alone[l[0].graph]) continue;  // that graph's own launch
      uint64_t v = 0, m = 0;
      size_t k = 0;
      for (const auto &pk : l) {
        v += gn[pk.graph], m += gm[pk.graph];
        if (pk.q.size() > k) k = pk.q.size();
      }
      if (v > need.max_v || m > need.max_m || v * union_row_width(k) > need.entries) puts("too small");
      if (l.size() > 1 && v * union_row_width(k) > p.entries) puts("entries");
    }
  }
  return 0;
}
"""


@pytest.mark.parametrize("seed", range(6))
def test_need_covers_every_plan(tmp_path, seed):
    (tmp_path / "n.cpp").write_text(DRIVER)
    exe = tmp_path / "n"
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", str(ROOT / "grus_framework_gb300" / "csrc"),
                    str(tmp_path / "n.cpp"), "-o", str(exe)], check=True)
    rng = np.random.default_rng(seed)
    text = []
    for _ in range(200):
        G, cap = int(rng.integers(1, 20)), int(2 ** rng.uniform(10, 24))
        n = (2 ** rng.uniform(2, 21, G)).astype(np.int64)
        m = (n * rng.uniform(0, 40, G)).astype(np.int64)
        alone = (rng.random(G) < 0.7) & (n * 8 <= cap)
        qg = np.sort(rng.integers(0, G, int(rng.integers(1, 300))))
        text.append(f"{G} {len(qg)} {cap} {int(rng.integers(1, 65))}")
        text += [f"{a} {b} {int(c)}" for a, b, c in zip(n, m, alone)]
        text.append(" ".join(map(str, qg)))
    out = subprocess.run([str(exe)], input="\n".join(text) + "\n", capture_output=True, text=True, check=True)
    assert out.stdout == ""
