"""The one-correction division of the SQA thresholds (acceptance in csrc/sb_sqa_tc.cuh): t = RN(a RN(1/b)), then
RN(t + (a - b t) RN(1/b)), both steps fused, is RN(a / b) for all significands a, b.

The value before the last rounding lies within 2^-22 ulp of a / b: t is off by less than 2 ulp, the remainder rounds by
at most 2^-24 of itself and the reciprocal is off by at most 2^-24. So only quotients closer than that to the midpoint
of two floats can round wrongly. With integer significands A, B in [2^23, 2^24) a midpoint is (2 q + 1) / 2 at the
quotient's scale, and A 2^S - B (2 q + 1) = r, S = 24 or 25, is the distance in units of 1 / (2 B) ulp: at least 1 and,
for the close ones, at most 2^-22 2 B < 8. All pairs with |r| <= 8 are enumerated (r fixes 2 q + 1 modulo a power of
two) and compared with the IEEE division. The exponents play no part: 2^-24 <= a < 17 and beta lies in [1/16, 8]."""
import os
import re
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include <math.h>
#include <stdint.h>
#include <stdio.h>
int main() {
  long pairs = 0, wrong = 0;
  for (uint32_t B = 1u << 23; B < 1u << 24; ++B) {
    const int k = __builtin_ctz(B);  // r has B's power of two
    const uint32_t odd = B >> k;
    uint32_t inv = odd;
    for (int i = 0; i < 5; ++i) inv *= 2 - odd * inv;
    const float b = (float)B, rb = 1.0f / b;
    for (int r = -8; r <= 8; ++r) {
      if (r == 0 || __builtin_ctz(r < 0 ? -r : r) != k) continue;
      for (int S = 24; S <= 25; ++S) {  // A >= B, A < B
        const uint32_t mod = 1u << (S - k);
        for (uint64_t m = (uint32_t)(-(r >> k)) * inv & (mod - 1); m < 1u << 25; m += mod) {
          if (m < 1u << 24 || !(m & 1)) continue;
          const int64_t A = ((int64_t)B * (int64_t)m + r) >> S;
          if (A < 1 << 23 || A >= 1 << 24 || (S == 24) != (A >= (int64_t)B)) continue;
          const float a = (float)A, t = a * rb;
          ++pairs;
          wrong += fmaf(fmaf(-b, t, a), rb, t) != a / b;
        }
      }
    }
  }
  printf("%ld %ld\n", pairs, wrong);
}
"""


def test_one_correction_is_the_ieee_quotient(tmp_path):
    code = open(os.path.join(ROOT, "annealing_gb300", "csrc", "sb_sqa_tc.cuh")).read()
    body = re.sub(r"\s+", " ", code[code.index("float acceptance("):])
    assert "t = __fmul_rn(a, rbeta); return u24 ? __fmaf_rn(__fmaf_rn(-beta, t, a), rbeta, t)" in body
    assert "rbeta = __frcp_rn(beta)" in re.sub(r"\s+", " ", code)
    src, exe = tmp_path / "div.c", tmp_path / "div"
    src.write_text(PROGRAM)
    subprocess.run(["gcc", "-O2", "-ffp-contract=off", "-fno-fast-math", str(src), "-o", str(exe), "-lm"], check=True)
    pairs, wrong = map(int, subprocess.run([str(exe)], stdout=subprocess.PIPE, text=True, check=True).stdout.split())
    assert pairs > 10_000_000 and wrong == 0
