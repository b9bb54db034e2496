"""From which length on pairs get a bound probe (bound_limits in tsu_plan.h):
the lines of the rule, and its host arithmetic against exact integers."""
import random
import subprocess

import pytest

from test_kernel_emu import EMU_DIR

SRC = r"""
#include "@EMU@/warp_emu.h"
#include "@EMU@/../../tsunami_pact_b200/csrc/tsu_plan.h"
#include <cstdio>
#include <cstdlib>
using namespace tsu;
int main(int argc, char** v) {
  auto a = [&](int i) { return std::atoll(v[i]); };
  int g = 1;
  const Pen p = a(2) < 0 ? reduce_linear((int)a(1), (int)a(3), &g) : reduce_penalties((int)a(1), (int)a(2), (int)a(3), (int)a(4), (int)a(5), &g);
  const BoundLimits b = bound_limits(p, 232448);
  std::printf("%d %d %d %d %d\n", b.side, b.few_side, p.go, p.ge, p.min_ge());
  for (int i = 6; i + 2 < argc; i += 3) {
    int lo, hi;
    bound_reach(p, (int)a(i), (int)a(i + 1), (int)a(i + 2), &lo, &hi);
    std::printf("%d %d\n", lo, hi);
  }
}
"""


@pytest.fixture(scope="module")
def rule(tmp_path_factory):
    d = tmp_path_factory.mktemp("rule")
    (d / "rule.cpp").write_text(SRC.replace("@EMU@", EMU_DIR))
    exe = str(d / "rule")
    subprocess.run(["g++", "-std=c++20", "-O2", "-w", "-o", exe, str(d / "rule.cpp"), "-lpthread"], check=True)

    def run(pen, pairs=()):
        o2, e2 = (pen[3], pen[4]) if len(pen) == 5 else (-1, 0)
        args = [str(x) for x in (*pen[:3], o2, e2)] + [str(x) for p in pairs for x in p]
        out = subprocess.run([exe] + args, capture_output=True, check=True, text=True).stdout.split("\n")
        return [[int(x) for x in ln.split()] for ln in out if ln]

    return run


def test_lines(rule):
    """The width at 4 % edits is 2 s / e for a score s of (dearest edit x edits)
    and 16; a hundred bases of slack around where it reaches the rule's."""
    for pen, want in (((4, 6, 2), 1212), ((3, 5, 1), 1024), ((1, -1, 1), 4850), ((4, 6, 2, 24, 1), 300), ((20, 30, 7), 519)):
        side = rule(pen)[0][0]
        assert abs(side - want) <= 2, (pen, side)


def test_reach_is_exact(rule):
    """Equal to integer arithmetic for lengths up to 2^26 and bounds up to 2^31."""
    rng = random.Random(3)
    for pen in ((4, 6, 2), (5, 60, 4), (3, 5, 1), (127, 60, 63)):
        pairs = []
        for _ in range(300):
            m = int(2 ** rng.uniform(0, 26))
            n = min(1 << 26, max(1, m + rng.choice([0, 1, -1, rng.randint(-m, m)])))
            pairs.append((m, n, rng.randint(0, int(2 ** rng.uniform(4, 30)))))
        out = rule(pen, pairs)
        go, ge, e = out[0][2:]

        def div(a, b):  # towards 0
            return abs(a) // b * (1 if a >= 0 else -1)

        def side(k, ub):
            s = div((k - 1) * ge * e + ub * ge + go * e, ge + e)
            return max(k, 0, 1 + div(s - go, ge) if s >= go else 0) + 2

        for (m, n, ub), (lo, hi) in zip(pairs, out[1:]):
            h, low = side(n - m, ub), side(m - n, ub)
            assert (lo, hi) == (-low if low < m else -m, h if h < n else n), (pen, m, n, ub)
