"""The ring arithmetic of the tcgen05 matvec's MMA warps (csrc/ring.h), compiled for the host and replayed over every ring depth
and items of odd and even length: slot and parity must be those of the chunk's number, and no step may go backwards."""
import subprocess
from pathlib import Path

CSRC = Path(__file__).resolve().parents[1] / "mlx-metal-kernels_b200" / "csrc"

DRIVER = r"""
#include "ring.h"
#include <cstdio>
using namespace b200q;

// the two loops of the MMA issuers in qgemm_ts.cu: two chunks per round of waits (two matrices), and one
template <int MATS> int replay(int j, int per, int items, int n_ch, int xs, int na) {
    ChunkWalk<MATS> w(j);
    int bad = 0, seen = 0, want = 0;
    auto look = [&](int g) {
        const int a = MATS * g + (MATS == 2 ? j : 0);
        bad += w.x.slot != g % xs || w.x.par != ((uint32_t)(g / xs) & 1u) || w.a.slot != a % na || w.a.par != ((uint32_t)(a / na) & 1u);
        ++seen;
    };
    for (int it = 0; it < items; ++it) {
        if (MATS == 2 && per == 2) {
            for (int ch = 0; ch < n_ch; ch += 2) {
                w.to(it * n_ch + ch, xs, na);
                look(it * n_ch + ch);
                const bool two = ch + 1 < n_ch;
                if (two) { w.to(it * n_ch + ch + 1, xs, na); look(it * n_ch + ch + 1); }
            }
        } else {
            for (int ch = ChunkWalk<MATS>::first(j); ch < n_ch; ch += 1 + ChunkWalk<MATS>::kSkip) {
                w.to(it * n_ch + ch, xs, na);
                look(it * n_ch + ch);
            }
        }
        want += MATS == 2 ? n_ch : (n_ch + 1 - j) / 2;
    }
    return bad + (seen != want);
}
int main() {
    int bad = 0, runs = 0;
    for (int n_ch = 1; n_ch <= 60; ++n_ch)
        for (int na = 2; na <= 8; na += 2)
            for (int j = 0; j < 2; ++j) {
                for (int xs = 2; xs <= 8; xs += 2, ++runs) bad += replay<1>(j, 1, 4, n_ch, xs, na);
                for (int xs = 2; xs <= 8; ++xs)
                    for (int per = 1; per <= 2; ++per, ++runs) bad += replay<2>(j, per, 4, n_ch, xs, na);
            }
    std::printf("%d %d\n", runs, bad);
    return 0;
}
"""


def test_slot_and_parity_follow_the_chunk_number(tmp_path):
    (tmp_path / "driver.cpp").write_text(DRIVER)
    subprocess.run(["g++", "-O1", "-std=c++17", f"-I{CSRC}", str(tmp_path / "driver.cpp"), "-o", str(tmp_path / "driver")], check=True)
    runs, bad = map(int, subprocess.run([str(tmp_path / "driver")], check=True, capture_output=True, text=True).stdout.split())
    assert runs > 1000 and bad == 0
