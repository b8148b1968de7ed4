"""The log-sum-exp form of the reproducible exponential (csrc/portable_math.h)
equals the general one bit for bit: around every rounding boundary of its
exponent, at the edges of its range, at random, and for special values."""
import pathlib
import shutil
import subprocess

import pytest

ROOT = pathlib.Path(__file__).resolve().parents[1]

SOURCE = r"""
#include <stdio.h>
#include "portable_math.h"
static long check(float x) {
  const uint32_t a = thmm_f2u(thmm_expf(x)), b = thmm_f2u(thmm_expf_nonpositive(x));
  if (a != b)
    printf("x = %a: %08x, %08x\n", x, a, b);
  return a != b;
}
int main(void) {
  long failures = 0;
  const float special[] = {0.0f, -0.0f, 1.0f, -87.0f, -103.9f, -104.0f, -1e30f,
                           thmm_u2f(0xff800000u), thmm_u2f(0x7fc00000u), -1e-45f};
  for (unsigned i = 0; i < sizeof special / sizeof *special; ++i)
    failures += check(special[i]);
  for (int half = 0; half <= 300; ++half) { /* x / ln 2 = -half / 2 */
    const uint32_t at = thmm_f2u(-0.5f * (float)half * 0.69314718f);
    for (int d = -64; d <= 64; ++d)
      failures += check(thmm_u2f(at + (uint32_t)d));
  }
  uint32_t state = 1;
  for (int i = 0; i < 4000000; ++i) {
    state = state * 1664525u + 1013904223u;
    failures += check(-110.0f * (float)(state >> 8) / 16777216.0f);
  }
  return failures != 0;
}
"""


def test_nonpositive_exponential_is_the_general_one(tmp_path):
    cc = shutil.which("gcc")
    if cc is None:
        pytest.skip("needs gcc")
    source = tmp_path / "paths.c"
    source.write_text(SOURCE)
    binary = tmp_path / "paths"
    subprocess.run([cc, "-std=c11", "-O2", "-ffp-contract=off",
                    f"-I{ROOT / 'parallel_tree_hmm_gb300' / 'csrc'}", str(source), "-o",
                    str(binary), "-lm"], check=True)
    result = subprocess.run([str(binary)], capture_output=True, text=True, timeout=300)
    assert result.returncode == 0, result.stdout[:2000]
