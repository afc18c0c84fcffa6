"""What belongs to a device is asked for once on each device, not once in a
process (csrc/cuda/fmdg_perdev.h)."""
import glob
import os
import re
import subprocess

CUDA = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "fmd_gb300", "csrc", "cuda")

PROGRAM = r"""
#include "fmdg_perdev.h"
#include <cstdio>

int main()
{
    static PerDevice kept;
    int asked[3] = {0, 0, 0};
    auto blocks = [&](int device) {
        return kept.get(device, [&] { asked[device]++; return device == 1 ? 8 : 16; });
    };
    const int a = blocks(0), b = blocks(1), c = blocks(0), d = blocks(1), e = blocks(2);
    int outside = 0;
    for (int k = 0; k < 2; k++) outside += kept.get(64, [] { return 3; }) + kept.get(-1, [] { return 4; });
    std::printf("%d %d %d %d %d asked %d %d %d outside %d", a, b, c, d, e, asked[0], asked[1], asked[2], outside);
    return 0;
}
"""


def test_asked_once_per_device(tmp_path):
    src, exe = tmp_path / "p.cc", tmp_path / "p"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-I" + CUDA, str(src), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout
    assert out == "16 8 16 8 16 asked 1 1 1 outside 14"


def test_no_answer_kept_for_the_process():
    """(a function-local static formed by a call would be the first device's
    answer for all of them)"""
    for path in glob.glob(os.path.join(CUDA, "*.cu*")):
        assert not re.search(r"static const int \w+ = \[", open(path).read()), path
