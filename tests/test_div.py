"""The branchless quotients of include/ice_div.h against the compiled division, on the host: the same bits for
random operands of the range they take, significands next to 1 and 2 and near-midpoint quotients included, from
a first reciprocal that is off by up to 2^-20 (what the device's instruction promises)."""
import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parents[1]
SRC = r'''
#include <stdio.h>
#include <stdint.h>
#include <string.h>
#include "ice_div.h"
static uint64_t s = 88172645463325252ull;
static uint64_t rn(void) { s ^= s << 13; s ^= s >> 7; s ^= s << 17; return s; }
static double mk(uint64_t m, int e) {
  uint64_t u = ((uint64_t)(1023 + e) << 52) | (m & 0xfffffffffffffull); double d; memcpy(&d, &u, 8); return d;
}
int main(void) {
  long bad = 0, n = 0;
  for (long i = 0; i < 4000000; ++i) {
    uint64_t ma = rn(), mb = rn(); int k = rn() % 6;
    if (k == 1 || k == 4) mb = ~(rn() >> (36 + rn() % 28));       /* significands next to 2 ... */
    if (k == 2) mb = rn() >> (36 + rn() % 28);                    /* ... and to 1 */
    if (k == 3) ma = ~(rn() >> (36 + rn() % 28));
    if (k == 4) ma = rn() >> (36 + rn() % 28);
    double a = mk(ma, (int)(rn() % 380) - 190), b = mk(mb, (int)(rn() % 380) - 190);
    if (k == 5) { double q = mk(rn(), 0); a = fma(0x1p-53 * q, b, q * b); }   /* next to a midpoint */
    if (rn() % 64 == 0) a = 0.0;
    if (rn() & 1) a = -a;
    if (rn() & 1) b = -b;
    if (!ice_div_by(b) || (a != 0.0 && !ice_div_in(a))) continue;
    double y0 = (1.0 / b) * (1.0 + (double)(int64_t)rn() / 9.3e18 * 0x1p-20);
    double q = ice_div_quot(a, b, ice_div_refine(b, y0));
    ++n;
    if (q != a / b) ++bad;
  }
  double out[] = {0x1p-201, 0x1p200, 1.0 / 0.0, 0.0 / 0.0, 0.0, 5e-324, 0x1.fffffffffffffp0};
  for (int i = 0; i < 7; ++i) if (ice_div_by(out[i])) ++bad;
  printf("%ld %ld\n", bad, n);
  return 0;
}
'''


def test_quotients_are_ieee(tmp_path):
    (tmp_path / "d.c").write_text(SRC)
    exe = tmp_path / "d"
    subprocess.run(["gcc", "-O2", "-ffp-contract=off", f"-I{ROOT / 'include'}", "-o", str(exe), str(tmp_path / "d.c"),
                    "-lm"], check=True)
    bad, n = (int(x) for x in subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.split())
    assert n > 3_000_000 and bad == 0
