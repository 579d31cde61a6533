"""The layouts pool members get (wendy_gb300/csrc/wg_layout.h, plain host code),
compiled here and checked over every size up to 1e5 sheets and every target a
step may ask for."""
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(__file__), "..", "wendy_gb300", "csrc")

PROGRAM = r"""
#include <cstdio>
#include <cstdlib>
#include "wg_layout.h"
using namespace wg;
int main(int argc, char** argv) {
  const int tuned = atoi(argv[1]);
  for (int64_t n = 1; n <= 100000; n += n < 20000 ? 1 : 7) {
    const int64_t nb_tuned = (n + tuned - 1) / tuned;
    int64_t room = (n + kMinTarget - 1) / kMinTarget;
    if (room > 1024) room = 1024;
    if (room < nb_tuned) room = nb_tuned;
    for (int64_t t = kMinTarget; t <= 1600; t += n < 8000 ? 1 : 32) {
      const MemberLayout l = member_layout(n, tuned, nb_tuned, room, t);
      // all sheets have a bucket, and no bucket is empty ...
      const bool cover = l.nb * l.target >= n && (l.nb - 1) * l.target < n;
      // ... a quarter of the slots or more is spare, as in the tuned layouts ...
      const bool spare = 3 * l.capg >= 4 * l.target && l.capg <= kBucketCap;
      // ... bulk copies of four sheets stay in place, and so do all buckets
      const bool fits = l.capg % 4 == 0 && l.nb * l.capg <= nb_tuned * kBucketCap &&
                        l.nb <= room && l.target <= tuned && l.target >= 1;
      if (!cover || !spare || !fits) {
        printf("n %ld t %ld: target %d nb %ld slots %d\n", (long)n, (long)t, l.target,
               (long)l.nb, l.capg);
        return 1;
      }
    }
  }
  return 0;
}
"""


@pytest.mark.parametrize("tuned", [64, 384, 700, 1024, 1280, 1536])
def test_every_bucket_has_spare_slots(tmp_path, tuned):
    src, exe = tmp_path / "layout.cpp", tmp_path / "layout"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O2", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe), str(tuned)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
