"""The branchless quotients of include/ice_div.h next to the midpoints of two doubles, on the host: for a divisor
of significand B (odd, 53 bits) the dividends whose quotients lie k / (2^54 B), k = 1 or 3, off a midpoint solve
2^54 A = B (2 Q + 1) +- k, so 2 Q + 1 is -+ k times the inverse of B modulo 2^54. Divisors next to 2, next to the
largest that ice_div_by takes and at random; first reciprocals at both ends of the error the header allows
(2^-20), at half of it and exact."""
import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parents[1]
SRC = r'''
#include <stdio.h>
#include <stdint.h>
#include <math.h>
#include "ice_div.h"
typedef unsigned __int128 u128;
static uint64_t s = 88172645463325252ull;
static uint64_t rn(void) { s ^= s << 13; s ^= s >> 7; s ^= s << 17; return s; }
static long bad, n, taken;
static void divisor(uint64_t B) {
  const uint64_t M = (1ull << 54) - 1;
  const double b = ldexp((double)B, -52);
  if (!ice_div_by(b)) return;
  ++taken;
  uint64_t x = B;                                    /* the inverse of B modulo 2^64, Newton */
  for (int i = 0; i < 6; ++i) x *= 2 - B * x;
  for (int k = -3; k <= 3; k += 2) {
    const uint64_t h = ((uint64_t)(int64_t)(-k) * x) & M;               /* 2 Q + 1 */
    if (h < (1ull << 53)) continue;
    const u128 t = (u128)B * h + (u128)(__int128)k;
    const uint64_t A = (uint64_t)(t >> 54);
    if ((t & M) || A < (1ull << 52) || A >= (1ull << 53)) continue;
    for (int e = -4; e <= 4; ++e) {
      const double a = ldexp((double)A, (int)(rn() % 60) - 30);
      const double y0 = (1.0 / b) * (1.0 + e * 0.25 * 0x1p-20);
      ++n;
      if (ice_div_quot(a, b, ice_div_refine(b, y0)) != a / b) ++bad;
    }
  }
}
int main(void) {
  for (uint64_t j = 1; j < 40000; j += 2) divisor((1ull << 53) - j);
  for (int e = 14; e < 53; ++e)                                 /* 2 - j 2^-52 on both sides of the proof's cases */
    for (uint64_t j = 1; j < 4000; j += 2) { divisor((1ull << 53) - (1ull << e) - j); divisor((1ull << 53) - (1ull << e) + j); }
  for (uint64_t j = 1; j < 40000; j += 2) divisor((1ull << 52) + j);
  for (int i = 0; i < 400000; ++i) divisor(((rn() >> 12) | (1ull << 52)) | 1);
  for (int i = 0; i < 400000; ++i) divisor(((1ull << 53) - (rn() >> (12 + rn() % 40))) | 1);
  printf("%ld %ld %ld\n", bad, n, taken);
  return 0;
}
'''


def test_quotients_next_to_midpoints(tmp_path):
    (tmp_path / "d.c").write_text(SRC)
    exe = tmp_path / "d"
    subprocess.run(["gcc", "-O2", "-ffp-contract=off", f"-I{ROOT / 'include'}", "-o", str(exe), str(tmp_path / "d.c"),
                    "-lm"], check=True)
    bad, n, taken = (int(x) for x in subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.split())
    assert taken > 400_000 and n > 4_000_000 and bad == 0, (bad, n, taken)
