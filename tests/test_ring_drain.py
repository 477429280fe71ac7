"""The drain of a ring of copies (csrc/ring_drain.h), compiled for the host and run on a model of the stages' mbarriers: after
it no copy is under way, and it waits for none that was never made."""
from __future__ import annotations

import os
import subprocess

PROGRAM = r"""
#include "ring_drain.h"
#include <cstdio>
#include <cstdlib>
#include <vector>

// A stage's barrier: phases armed and completed. A wait for parity x returns at once where the phase before the current one has
// that parity (or none has: the phase "before the first" has parity 1), else when the current one completes.
struct Barrier { int armed = 0, done = 0; };
static int run(int stages, int chunks, int stopped) {
    std::vector<Barrier> full(stages);
    auto bring = [&](int c) { if (c < chunks) full[c % stages].armed++; };
    auto wait = [&](int s, unsigned parity) {
        Barrier& b = full[s];
        if (((unsigned)b.done & 1u) != parity) return;         // (the phase it names lies behind)
        if (b.armed == b.done) { std::printf("waits for a copy that was never made\n"); std::exit(1); }
        b.done++;
    };
    for (int s = 0; s < stages; ++s) bring(s);
    for (int i = 0; i < stopped; ++i) {
        wait(i % stages, (unsigned)(i / stages) & 1u);
        bring(i + stages);
    }
    const int brought = stopped + stages < chunks ? stopped + stages : chunks;
    celeg_b200::drain_ring(stopped, brought, stages, wait);
    for (const Barrier& b : full)
        if (b.armed != b.done) return 1;
    return 0;
}
int main() {
    for (int stages = 1; stages <= 4; ++stages)
        for (int chunks = 1; chunks <= 13; ++chunks)
            for (int stopped = 0; stopped <= chunks; ++stopped)
                if (run(stages, chunks, stopped)) { std::printf("%d stages, %d chunks, stopped at %d\n", stages, chunks, stopped); return 1; }
    return 0;
}
"""


def test_every_copy_under_way_is_waited_for(tmp_path):
    source, program = tmp_path / "drain.cpp", tmp_path / "drain"
    source.write_text(PROGRAM)
    csrc = os.path.join(os.path.dirname(os.path.abspath(__file__)), os.pardir, "celeg_b200", "csrc")
    subprocess.run(["g++", "-std=c++17", "-I", csrc, str(source), "-o", str(program)], check=True)
    result = subprocess.run([str(program)], stdout=subprocess.PIPE, text=True)
    assert result.returncode == 0, result.stdout
