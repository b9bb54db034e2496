"""Low-memory mode with an interval: the rungs its passes start from and climb
to, which set how wide its checkpoints are."""
import ctypes
import subprocess

import numpy as np
import pytest

from test_kernel_emu import EMU_DIR

SRC = r"""
#include "@EMU@/warp_emu.h"
#include "@EMU@/../../tsunami_pact_b200/csrc/tsu_plan.h"
#include <cstdio>
using namespace tsu;
int main() {
  int g = 1;
  const Pen p = reduce_penalties(4, 6, 2, -1, 0, &g);
  auto next = [&](int gw, int side, bool low) {
    const PassChoice c = next_pass({kModeShared, gw}, p, side, side, 232448, 16, low);
    std::printf("%d %d %d\n", c.mode, c.gw, c.single ? 1 : 0);
  };
  next(16, 16370, true);   // the shared ring has had it: the global one
  next(16, 16370, false);  // handed back by the packed kernel for its length
  next(16, 20000, true);
  next(8, 16370, true);
  // a ring of all m + n + 3 diagonals on the fewest warps that hold it
  const int w = shared_ring_width(p, 2, 2 * (2 * (int)packed_words(500)), 232448, false);
  next(1, (w - 3) / 2, true);
  std::printf("%d %d\n", w, shared_ring_width(p, 2, 2 * (2 * (int)packed_words(500)), 232448, true));
}
"""


def test_ladder(tmp_path):
    (tmp_path / "low.cpp").write_text(SRC.replace("@EMU@", EMU_DIR))
    exe = str(tmp_path / "low")
    subprocess.run(["g++", "-std=c++20", "-O1", "-w", "-o", exe, str(tmp_path / "low.cpp"), "-lpthread"], check=True)
    out = subprocess.run([exe], capture_output=True, check=True, text=True).stdout.split("\n")
    assert out[:4] == ["1 16 0", "0 16 1", "1 16 0", "0 16 0"]
    assert out[4] == "0 2 0"
    low, packed = map(int, out[5].split())
    assert low > packed  # (its rows have no row of absent cells beside them)


@pytest.mark.gpu
@pytest.mark.parametrize("pairs, length", [(1, 900), (30, 900), (1, 8000), (30, 8000), (1, 16370)])
def test_few_pairs_keep_the_rung(oracle, pairs, length):
    """Few pairs hold what the compiled rung holds (one 8 kbp pair with
    checkpoints every 50 scores: 12 MB on 8 warps, 32 on 16)."""
    import tsunami_pact_b200 as T

    b = T.gen_batch(7, np.full(pairs, length, np.int32), np.full(pairs, 0.05))
    pats = [bytes(b[0][b[1][i]:b[1][i] + b[2][i]]) for i in range(pairs)]
    txts = [bytes(b[3][b[4][i]:b[4][i] + b[5][i]]) for i in range(pairs)]
    osc, oops = oracle.align_batch(pats, txts, 4, 6, 2)
    L = T.lib()
    L.tsu_set_band_start.argtypes = [ctypes.c_void_p] + [ctypes.c_int] * 3
    L.tsu_get_band_start.argtypes = [ctypes.c_void_p, ctypes.c_int] + [ctypes.POINTER(ctypes.c_int)] * 2
    held, logs = [], []
    for as_compiled in (False, True):
        with T.Aligner(4, 6, 2) as al:
            al.set_low_memory(50)
            for band in range(6):
                m, w = ctypes.c_int(), ctypes.c_int()
                assert L.tsu_get_band_start(al._h, band, ctypes.byref(m), ctypes.byref(w)) == 0
                if as_compiled:
                    assert L.tsu_set_band_start(al._h, band, m.value, w.value) == 0
            scores, ops = al.align(pats, txts)
            assert list(scores) == list(osc) and ops == oops
            held.append(al.timing()["device_bytes"])
            logs.append([p.split("@")[0] for p in al.pass_log().split()])
    assert held[0] == held[1] and logs[0] == logs[1], (held, logs)
    assert len(set(logs[0])) == len(logs[0]), logs[0]  # no rung twice
