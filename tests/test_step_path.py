"""The rule that picks the kernels of a pass (csrc/step_path.h, plain C++), compiled and evaluated on the host."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "espresso_b200", "csrc")
MAIN = r"""
#include <cstdio>
#include "step_path.h"
int main() {
    for (int r = 1; r < 5000; r++)
        if (esp::slot_row_words(r) % 4 || esp::slot_row_words(r) < 6ull * r) return 1;  // the lists behind it hold 16-byte elements
    int ready, quantised, tp, d, rows;
    while (scanf("%d %d %d %d %d", &ready, &quantised, &tp, &d, &rows) == 5) printf("%d\n", (int)esp::step_path(ready, quantised, tp, d, rows));
}
"""
ROWWISE, STREAM, TILES, REFUSED = range(4)


@pytest.fixture(scope="module")
def path(tmp_path_factory):
    gxx = shutil.which("g++")
    if not gxx:
        pytest.skip("no g++")
    d = tmp_path_factory.mktemp("step_path")
    (d / "main.cc").write_text(MAIN)
    subprocess.run([gxx, "-std=c++17", "-I", CSRC, "-o", str(d / "main"), str(d / "main.cc")], check=True)

    def ask(ready, quantised, tp, d_model, rows):
        line = f"{ready} {quantised} {tp} {d_model} {rows}\n"
        return int(subprocess.run([str(d / "main")], input=line, capture_output=True, text=True, check=True).stdout)

    return ask


@pytest.mark.parametrize("quantised", [0, 1])
@pytest.mark.parametrize("rows", [1, 2, 8, 64, 65, 704, 705, 2048])
def test_tensor_parallel_ranks_never_take_the_rowwise_kernels(path, quantised, rows):
    """Only the batched paths add up the ranks' partial sums and know the vocabulary shard."""
    for d_model in (256, 2048, 4096):
        assert path(1, quantised, 2, d_model, rows) in (STREAM, TILES)
        assert path(0, quantised, 2, d_model, rows) == REFUSED


def test_single_device_rows(path):
    assert path(1, 1, 1, 2048, 1) == ROWWISE and path(1, 1, 1, 2048, 2) == STREAM  # a quantised row reads the blocks
    assert path(1, 0, 1, 2048, 1) == STREAM
    assert path(0, 0, 1, 2048, 300) == ROWWISE
    for d_model, rows in ((768, 704), (2048, 192), (4096, 64)):
        assert path(1, 0, 1, d_model, rows) == STREAM and path(1, 0, 1, d_model, rows + 1) == TILES
