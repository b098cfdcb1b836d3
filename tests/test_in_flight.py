"""Which memory a kernel may read before it has waited for the kernel in front (csrc/in_flight.h), without a GPU."""
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "nuvec_b200" / "csrc"

# A stream as a list of launches; `early(p)`: may the next kernel read the 16 bytes at p before its wait?
PRELUDE = r"""
#include "in_flight.h"
#include <cassert>
using namespace nvc;
static char mem[1 << 16];
static InFlight w;
[[maybe_unused]] static Writes at(Trigger t, int p, size_t n = 16) { return Writes(t, {{mem + p, n}}); }
[[maybe_unused]] static void launch(const Writes &x) { w.note(x, w.room(x)); }
[[maybe_unused]] static bool early(int p, size_t n = 16) { return w.clear_of(mem + p, n); }
constexpr Trigger EARLY = Trigger::EARLY, LATE = Trigger::LATE;
"""

CASES = {
    # the kernel directly in front wrote it, whether that one triggers or not: its stores show behind the wait only
    "directly in front": "launch(at(LATE, 0)); assert(!early(0) && early(16)); launch(at(EARLY, 32)); assert(!early(32));",
    # a kernel that waits before it triggers ends everything in front of it, one that triggers first does not
    "further in front": "launch(at(LATE, 0)); launch(at(EARLY, 64)); launch(at(EARLY, 128)); assert(!early(0) && !early(64));"
                        "launch(at(LATE, 192)); assert(early(0) && early(64) && early(128) && !early(192));",
    "edges": "launch(at(LATE, 32)); assert(early(16) && early(48) && !early(31, 2) && !early(47, 1) && !early(0, 4096));",
    "launch without a note": "w.unknown(); assert(!early(0)); launch(at(EARLY, 64)); assert(!early(0)); launch(at(LATE, 64)); assert(early(0) && !early(64));",
    "plain order": "launch(at(EARLY, 0)); w.note(at(EARLY, 64), false); assert(early(0) && !early(64));",
    "idle stream": "launch(at(EARLY, 0)); w.unknown(); w.finished(); assert(early(0));",
    "nothing written": "launch(Writes(EARLY, {})); launch(Writes(EARLY, {{nullptr, 16}, {mem, 0}})); assert(early(0));",
    # more distinct ranges than are kept: the launch without room goes in plain order, and nothing is forgotten before it
    "full": "int i = 0; while (w.room(at(EARLY, 16 * i))) { launch(at(EARLY, 16 * i)); assert(!early(0)); i++; } assert(i > 8);"
            "launch(at(EARLY, 16 * i)); assert(early(0) && !early(16 * i) && w.room(at(EARLY, 0)));",
    "the same blocks again": "for (int i = 0; i < 1000; i++) { assert(w.room(at(EARLY, 0))); launch(at(EARLY, 64 * (i % 7))); launch(at(EARLY, 0, 64)); }"
                             "assert(!early(0) && !early(48) && !early(384) && early(512));",
    "too many ranges": "Writes six(LATE, {{mem, 1}, {mem, 1}, {mem, 1}, {mem, 1}, {mem, 1}, {mem + 999, 1}}); assert(!w.room(six)); launch(six); assert(!early(999, 1));",
}


@pytest.mark.parametrize("name", CASES)
def test_window(name, tmp_path):
    (tmp_path / "t.cpp").write_text(PRELUDE + "int main() {" + CASES[name] + "}\n")
    subprocess.run(["g++", "-std=c++17", "-Wall", "-Werror", f"-I{CSRC}", "t.cpp", "-o", "t"], cwd=tmp_path, check=True)
    done = subprocess.run(["./t"], cwd=tmp_path, capture_output=True, text=True)
    assert done.returncode == 0, done.stderr
