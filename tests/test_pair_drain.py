"""How the product on SM pairs leaves after a wait gave up (csrc/pair_drain.h, plain C++), against a model of the barriers."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "espresso_b200", "csrc")
# A barrier of one arrival: a phase completes when the arrival is in and the byte count is zero.  Every copy that was issued
# lands late, after the drain has begun, one at a time; a phase that the drain waits for must not complete before the last copy
# of its fill, and must complete then.
MAIN = r"""
#include <cstdio>
#include <cstdlib>
#include <vector>
#include "pair_drain.h"
using namespace esp;
const int S = 5, B = 100;
struct Bar {
    int phase = 0, pending = 1; long tx = 0;
    void settle() { if (pending == 0 && tx == 0) { phase++; pending = 1; } }
    void expect(int b) { tx += b; if (pending == 0) abort(); pending--; settle(); }
    void land(int b) { tx -= b; settle(); }
    bool done(unsigned parity) const { return (phase & 1) != (int)parity; }
};
int main() {
    int cases = 0;
    for (int consumed = 0; consumed <= 13; consumed++)
        for (int n0 = consumed; n0 <= consumed + S; n0++)
            for (int n1 = consumed; n1 <= consumed + S; n1++) {
                Bar bar[S];
                for (int f = 0; f < consumed; f++) { bar[f % S].expect(2 * B); bar[f % S].land(B); bar[f % S].land(B); if (bar[f % S].phase != f / S + 1) return 1; }
                for (int f = consumed; f < n0; f++) bar[f % S].expect(2 * B);  // issued, in flight
                for (int f = pg_drain_begin(n0, n1, S); f < pg_drain_end(n0, n1); f++) {
                    const PgDrainStep d = pg_drain_step(f, n0, n1, S, B);
                    Bar& b = bar[d.stage];
                    if (d.expect) b.expect(d.expect);
                    if (d.complete) b.land(d.complete);
                    int flying = f < consumed ? 0 : (f < n0) + (f < n1);
                    while (flying--) { if (b.done(d.parity)) return 2; b.land(B); }
                    if (!b.done(d.parity)) return 3;
                }
                for (int s = 0; s < S; s++) if (bar[s].tx) return 4;
                cases++;
            }
    printf("%d\n", cases);
    return 0;
}
"""


def test_drain_waits_for_every_copy(tmp_path):
    gxx = shutil.which("g++")
    if not gxx:
        pytest.skip("no g++")
    (tmp_path / "main.cc").write_text(MAIN)
    subprocess.run([gxx, "-std=c++17", "-I", CSRC, "-o", str(tmp_path / "main"), str(tmp_path / "main.cc")], check=True)
    res = subprocess.run([str(tmp_path / "main")], capture_output=True, text=True)
    assert res.returncode == 0 and int(res.stdout) == 14 * 36
