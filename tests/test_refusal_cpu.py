"""Refused optional allocations (csrc/refusal.h): asked for again for less memory, or
after a number of frames, and not in every frame."""
import os
import shutil
import subprocess

import pytest

from conftest import PKG

PROGRAM = r"""
#include "refusal.h"
#include <cstdio>
// Frames that want `bytes`; returns how many of them ask while `free` bytes are there.
static int asks(cr::Refusal& r, int frames, size_t bytes, size_t free, bool* have) {
    int n = 0;
    for (int k = 0; k < frames && !*have; ++k) {
        if (r.stands(bytes)) continue;
        ++n;
        if (bytes <= free) *have = true;
        else r.refused(bytes);
    }
    return n;
}
int main() {
    cr::Refusal r;
    bool big = false, small = false;
    printf("%d ", asks(r, 1, 100, 50, &big));                          // the first frame asks
    printf("%d ", asks(r, cr::Refusal::kEvery - 1, 100, 50, &big));    // the next ones do not
    printf("%d ", asks(r, 1, 40, 50, &small));                         // a smaller request does, and is met
    printf("%d ", (int)small);
    printf("%d ", asks(r, 10 * cr::Refusal::kEvery, 100, 50, &big));   // one frame in kEvery
    printf("%d ", asks(r, cr::Refusal::kEvery, 100, 200, &big));       // memory is back
    printf("%d\n", (int)big);
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="no C++ compiler")
def test_refused_memory_is_asked_for_again(tmp_path):
    src = tmp_path / "refusal.cpp"
    src.write_text(PROGRAM)
    exe = tmp_path / "refusal"
    subprocess.run(["g++", "-std=c++17", "-Wall", "-Werror", "-I", os.path.join(PKG, "csrc"), str(src), "-o", str(exe)],
                   check=True)
    assert subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.split() == \
        ["1", "0", "1", "1", "10", "1", "1"]
