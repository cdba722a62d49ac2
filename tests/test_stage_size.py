"""The stage size of the record kernel's shared-memory ring (lgb_stage_floats of lagrbf_gb300/csrc/lgb_internal.h) for every
unit that the dispatcher chooses and any value of LAGRBF_TMA_BUDGET: stages on 16-byte boundaries, the ring within
shared memory, room for the final sums of the shares; and the measured sizes unchanged."""
import os
import subprocess

import lagrbf_gb300

CSRC = os.path.join(os.path.dirname(lagrbf_gb300.__file__), "csrc")

SOURCE = r"""
#include <stdio.h>
#include "lgb_internal.h"
#include "lgb_eval_tune.h"
int main(void)
{
  const int units[][2] = {{32, 32}, {64, 64}, {128, 128}, {128, 192}, {128, 256}, {256, 128}, {512, 128}}; /* threads, particles */
  long bad = 0;
  for (int u = 0; u < 7; u++)
    for (int nb = 2; nb <= 4; nb++)
      for (long long base = 256; base < 3000000; base += base < 20000 ? 1 : 99991) {
        const int t = units[u][0], b = lgb_stage_floats(base, nb, t, units[u][1]);
        bad += b % 4 != 0 || b < 32 || b > 1 << 14;
        bad += nb * (long)b * 4 + 2 * 128 * 16 * 4 + 512 * 16 * 4 + 8192 > 227 * 1024; /* ring, words per thread, static */
        bad += nb * (long)b < 6L * t;
      }
  printf("%ld %d %d %d %d %d %d\n", bad, lgb_stage_floats(LGB_TMA_BUDGET_TUNED, 2, 32, 32),
         lgb_stage_floats(LGB_TMA_BUDGET_TUNED, 2, 64, 64), lgb_stage_floats(LGB_TMA_BUDGET_TUNED, 2, 128, 128),
         lgb_stage_floats(LGB_TMA_BUDGET_TUNED, 2, 128, 256), lgb_stage_floats(LGB_TMA_BUDGET_TUNED, 2, 256, 128),
         lgb_stage_floats(LGB_TMA_BUDGET_TUNED, 2, 512, 128));
  return 0;
}
"""


def test_stage_sizes(tmp_path):
    src = tmp_path / "stage.c"
    src.write_text(SOURCE)
    subprocess.run(["gcc", "-O2", "-std=gnu11", "-I", CSRC, str(src), "-o", str(tmp_path / "stage")], check=True)
    out = subprocess.run([str(tmp_path / "stage")], check=True, stdout=subprocess.PIPE, text=True).stdout.split()
    assert list(map(int, out)) == [0, 512, 1024, 2048, 4096, 8192, 16384]
