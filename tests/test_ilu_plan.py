"""The rules that send block ILU substitutions to a thread-block cluster, compiled
for the host and checked around every limit: what the plan says fits does fit the
CTA's shared memory, with and without copies of other CTAs' rows, and FP64
substitutions are planned by one decision only. (The launch once had a bound of
its own, 32 bytes wider: without copies, 442,369 to 442,416 rows of one component
on 16 CTAs were launched in FP64 although no FP64 factors had been packed.)"""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SOURCE = r"""
#include "gb_ilu_plan.cuh"
#include <cstdio>
using namespace gb;

int main()
{
  long refused = 0, between = 0;
  for (int most = 8; most <= 16; most += 8)
    for (int B = 1; B <= 4; ++B)
      for (int size = 4; size <= 8; size += 4) {
        const int64_t limit = int64_t(kIluClusterBytes) / (B * size) * most;
        for (int64_t n = limit - 200; n <= limit + 200; ++n) {
          const IluPlan P = ilu_plan(n, B, 100, most);
          if (!P.ctas) {
            if (size == 8) { printf("n %ld B %d: fits FP32\n", long(n), B); return 1; }
            ++refused;
            continue;
          }
          if (int64_t(P.ctas) * P.chunk < n || P.ctas > most) {
            printf("n %ld B %d: rows left out\n", long(n), B);
            return 1;
          }
          // rows and zeros, as launched without copies
          const size_t places = (size_t(P.chunk) + 1) * B;
          if (places * P.value_bytes() > kIluClusterBytes + kIluZeroBytes) {
            printf("n %ld B %d: does not fit\n", long(n), B);
            return 1;
          }
          if (P.fp64 != (size_t(P.chunk) * B * 8 <= kIluClusterBytes)) {
            printf("n %ld B %d: fp64 %d\n", long(n), B, int(P.fp64));
            return 1;
          }
          between += !P.fp64 && places * 8 <= kIluClusterBytes + kIluZeroBytes;
          // the most copies that fit, and one more
          int64_t copies = 0;
          while (ilu_copies_fit(P, B, copies + 1))
            ++copies;
          if (copies && (size_t(P.chunk) + 1 + copies) * B * P.value_bytes() > kIluClusterBytes)
            return 1;
        }
      }
  printf("refused %ld between %ld\n", refused, between);
  return refused > 0 && between > 0 ? 0 : 1;
}
"""


def _run(tmp_path, source):
    gxx = shutil.which("g++")
    if not gxx:
        pytest.skip("no host compiler")
    src, exe = tmp_path / "t.cc", tmp_path / "t"
    src.write_text(source)
    subprocess.run([gxx, "-std=c++17", "-Wall", "-Werror", "-I",
                    os.path.join(ROOT, "gascoignelib_b200", "csrc"), "-o", str(exe), str(src)],
                   check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout


def test_plan_at_its_limits(tmp_path):
    _run(tmp_path, SOURCE)


PADDING = r"""
#include "gb_ilu_plan.cuh"
#include <cstdio>
using namespace gb;

// slots of n rows with `lower` and `upper` entries each, `per` rows of a level in a
// CTA, rounded up to groups of 32 rows and chunks of 8 entries
static int64_t slots(int64_t n, int per, int lower, int upper)
{
  const int64_t groups = (n + per - 1) / per * ((per + 31) / 32);
  return groups * 32 * ((lower + 7) / 8 * 8 + (upper + 7) / 8 * 8);
}

int main()
{
  auto ok = [](int64_t n, int per, int half) {
    const IluPlan P = ilu_plan(n, 1, int(n / per / 16 + 1), 16);
    return P.ctas > 0 && ilu_padding_ok(P, 1, slots(n, per, half, half), n * (2 * half + 1));
  };
  const bool r[] = {
    ok(274625, 38, 13),   // 65^3 rows, 27 entries
    ok(422500, 13, 4),    // 650^2 rows, 9 entries
    ok(400000, 6, 4),     // 200 x 2000 rows, numbered along the short side
    ok(4000, 1, 1),       // a short chain
    !ok(100000, 1, 1),    // a long one
    !ok(880000, 1, 1),    // and the longest that fits, in FP32
  };
  for (size_t k = 0; k < sizeof r; ++k)
    if (!r[k]) { printf("rule %zu\n", k); return 1; }
  return 0;
}
"""


def test_padding_rule(tmp_path):
    _run(tmp_path, PADDING)
