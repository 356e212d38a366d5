"""CPU: the words by which the one-cluster kernel's threads agree on what comes
next (grus_framework_gb300/csrc/narrow_steps.h), compiled with g++.  A thread
may read them late, when other CTAs are already a step ahead or other warps are
already pushing: what it reads must not depend on that, or threads of one block
go to different barriers."""
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]
DRIVER = r"""
#include <cstdio>
#include <cstring>
#include <initializer_list>
#include "narrow_steps.h"
using namespace grus::narrow;
static int fail(const char *what, unsigned step) {
  printf("%s at step %u\n", what, step);
  return 1;
}
// A fast CTA is past step `step` and has written the words of step + 1 (which
// it may do before a slow thread reads those of `step`).
int late_reads() {
  for (unsigned history = 0; history < 64; ++history) {
    StepWords w[2] = {};
    for (unsigned step = 1; step <= 6; ++step) {
      const bool sp = history >> (step - 1) & 1u, work = step % 3 != 0;
      if (sp) words_of(w, step).spilled = step;
      if (work) words_of(w, step).work = step;
      if (sp && work) words_of(w, step).late = step;
      StepWords ahead[2];
      memcpy(ahead, w, sizeof(w));
      words_of(ahead, step + 1).spilled = step + 1;
      words_of(ahead, step + 1).work = step + 1;
      words_of(ahead, step + 1).late = step + 1;
      for (const StepWords *v : {&words_of(w, step), &words_of(ahead, step)}) {
        if (found(v->spilled, step) != sp) return fail("spilled", step);
        if (found(v->work, step) != work) return fail("work", step);
        if (found(v->late, step) != (sp && work)) return fail("late", step);
      }
    }
  }
  return 0;
}
// Warps that reach the decision before a round at different times: the fastest
// has pushed `extra` entries in that round already, the slowest none.  Counts
// start anew in every step.
int late_warps() {
  for (unsigned own : {0u, 1u, 7u, 64u, 2048u})
    for (unsigned before : {0u, 3u, 29u, 300u, 9000u})
      for (unsigned extra : {1u, 30u, 100000u})
        for (unsigned step = 1; step <= 4; ++step)
          for (int round = 0; round < kRounds; ++round) {
            AwayCounts slow{}, fast{};
            for (int r = 0; r < round; ++r)
              away_in(slow, step, r) = away_in(fast, step, r) = before + r;
            away_in(fast, step, round) += extra;
            const bool go[2] = {goes_on(slow, step, round, own), goes_on(fast, step, round, own)};
            if (go[0] != go[1]) return fail("go on", step);
            if (round == 0 && !go[0]) return fail("first round", step);
            if (&away_in(fast, step, round) == &away_in(fast, step + 1, round))
              return fail("neighbouring steps share a count", step);
          }
  return 0;
}
"""


@pytest.fixture(scope="module")
def driver(tmp_path_factory):
    d = tmp_path_factory.mktemp("steps")
    (d / "steps.cpp").write_text(DRIVER + """
int main(int argc, char **argv) {
  if (argc > 1 && !strcmp(argv[1], "late_reads")) return late_reads();
  return argc > 1 && !strcmp(argv[1], "late_warps") ? late_warps() : 2;
}
""")
    exe = d / "steps"
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", str(ROOT / "grus_framework_gb300" / "csrc"),
                    str(d / "steps.cpp"), "-o", str(exe)], check=True)
    return exe


def test_step_words_read_late(driver):
    r = subprocess.run([str(driver), "late_reads"], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout


def test_rounds_decided_late(driver):
    r = subprocess.run([str(driver), "late_warps"], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
