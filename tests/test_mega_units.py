"""The units a load batch of the persistent kernels reads (csrc/mega_units.h, plain C++), compiled and checked on the host."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "espresso_b200", "csrc")
# Every warp (of 8, each with the units that are its own modulo 8, or alone) over chunks of every length, in batches of 2 to 8.
MAIN = r"""
#include <cstdio>
#include <initializer_list>
#include "mega_units.h"
int main() {
    for (int step : {1, 8})
        for (int batch : {2, 4, 6, 8})
            for (int nu = 1; nu < 200; nu++)
                for (int first = 0; first < step; first++) {
                    int next = first;  // the unit that the products must take next
                    for (int i0 = first; i0 < nu; i0 += step * batch)
                        for (int x = 0; x < batch; x++) {
                            const int i = esp::mega_batch_unit(i0, x, step, nu);
                            if (i < 0 || i >= nu || (i - first) % step) return 1;  // another warp's unit, or none of the chunk
                            if (i0 + x * step < nu) {
                                if (i != next) return 2;
                                next += step;
                            }
                        }
                    if (next < nu) return 3;
                }
    printf("ok\n");
}
"""


def test_a_batch_reads_units_of_its_own_warp(tmp_path):
    gxx = shutil.which("g++")
    if not gxx:
        pytest.skip("no g++")
    (tmp_path / "main.cc").write_text(MAIN)
    subprocess.run([gxx, "-std=c++17", "-I", CSRC, "-o", str(tmp_path / "main"), str(tmp_path / "main.cc")], check=True)
    res = subprocess.run([str(tmp_path / "main")], capture_output=True, text=True)
    assert res.returncode == 0 and res.stdout == "ok\n"
