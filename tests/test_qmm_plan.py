"""The plan of the many-row products (csrc/qmm_plan.h), without a GPU: which tile a shape takes, and that a schedule covers its tiles.

SHAPES is what the GPU tests rely on to reach every instantiation: rows, weight rows, inner size -> token tile, block pairs, at
148 multiprocessors and every bit width.
"""
import subprocess
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "nuvec_b200" / "csrc"
SHAPES = {(9, 130, 192): (32, False), (300, 520, 2176): (64, False), (65, 9490, 320): (128, False), (135, 9490, 192): (160, False),
          (2100, 2440, 64): (160, False), (163, 9490, 320): (192, False), (772, 4680, 320): (256, False), (198, 9490, 192): (256, True),
          (1601, 2460, 1088): (256, True), (2048, 12288, 4096): (256, True)}

PROGRAM = r"""
#include <cstdio>
#include <cstdlib>
#include <initializer_list>
#include "qmm_plan.h"
using namespace nvc;
int main(int argc, char **argv) {
    for (int i = 1; i + 3 < argc; i += 4) {
        const QmmPlan p = qmm_plan(atoll(argv[i]), 0, atoll(argv[i + 1]), atoi(argv[i + 2]) / QMM_BK, atoi(argv[i + 3]), 148);
        printf("%d %d\n", p.bt, (int)p.pair);
    }
    // every schedule: whole waves, then parts of whole tiles in at most two rounds of the workers, none of them empty
    for (int tiles = 1; tiles < 700; tiles++)
        for (int workers : {1, 74, 148})
            for (int kblocks : {1, 3, 8, 21, 64, 172})
                for (int grain : {4, 8})
                    for (int tokens : {9, 256}) {
                        float ns = -1.0f;
                        const Schedule s = make_schedule(tiles, workers, kblocks, grain, tokens, 300.0f, &ns);
                        const int grains = (kblocks + grain - 1) / grain, parts = s.tail_tiles * s.splits;
                        if (s.full_waves * workers + s.tail_tiles != tiles || s.tail_tiles >= workers || s.splits < 1 || s.splits > 16 || s.splits > grains ||
                            s.tail_rounds > 2 || (s.tail_tiles && (parts > s.tail_rounds * workers || parts <= (s.tail_rounds - 1) * workers)) || !(ns > 0.0f)) {
                            fprintf(stderr, "%d tiles, %d workers, %d blocks\n", tiles, workers, kblocks);
                            return 1;
                        }
                    }
    return 0;
}
"""


def test_plans_and_schedules(tmp_path):
    (tmp_path / "t.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-Wall", "-O1", f"-I{CSRC}", "t.cpp", "-o", "t"], cwd=tmp_path, check=True)
    asked = [(*shape, bits) for shape in SHAPES for bits in (2, 3, 4, 6, 8)]
    done = subprocess.run(["./t", *(str(v) for a in asked for v in a)], cwd=tmp_path, capture_output=True, text=True)
    assert done.returncode == 0, done.stderr
    got = [(int(bt), pair == "1") for bt, pair in (line.split() for line in done.stdout.splitlines())]
    for shape, plan in zip(asked, got):
        assert plan == SHAPES[shape[:3]], shape
    assert {p for p in got} == {(32, False), (64, False), (128, False), (160, False), (192, False), (256, False), (256, True)}
