"""The streaming line of AUTO support calls (csrc/support_rule.h) on the CPU, against calls timed both ways on a
GB300 (transactions, rows, candidates, us streamed, us staged; candidates of 2..8 items over sparse and over
sensor rows): the side it takes is never more than a tenth slower than the other."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "20261008-self-growing-evidence-agent_gb300", "csrc")

PROGRAM = r"""
#include <cstdio>
#include "support_rule.h"

int main() {
    const double t[][5] = {
         {5000, 77, 50000, 33, 37}, {5000, 77, 100000, 57, 42}, {5000, 77, 129999, 70, 45},
         {20000, 77, 50000, 51, 75}, {20000, 77, 100000, 91, 93}, {20000, 77, 129999, 115, 105},
         {20000, 1400, 50000, 55, 122}, {20000, 1400, 100000, 98, 144}, {20000, 1400, 279999, 248, 221},
         {5000, 640, 50000, 34, 42}, {5000, 640, 100000, 60, 46}, {5000, 640, 189999, 102, 58},
         {1048576, 640, 50000, 1407, 3525}, {1048576, 640, 100000, 2752, 4540}, {1048576, 640, 189999, 5102, 6488},
         {1048576, 1400, 50000, 1874, 4967}, {1048576, 1400, 100000, 3712, 5988}, {1048576, 1400, 279999, 10220, 9698},
         {1048576, 640, 50000, 1690, 3452}, {1048576, 640, 100000, 3267, 4374}, {1048576, 640, 189999, 6036, 6066},
         {2097152, 640, 50000, 3640, 7020}, {2097152, 640, 100000, 7114, 9049}, {2097152, 640, 189999, 13275, 12943},
         {4194304, 640, 50000, 8917, 14011}, {4194304, 640, 100000, 17458, 18070}, {4194304, 640, 189999, 33036, 25855},
         {4194304, 640, 50000, 11745, 13726}, {4194304, 640, 100000, 23095, 17407}, {4194304, 640, 189999, 43971, 24178},
         {16777216, 640, 50000, 43694, 55959}, {16777216, 640, 100000, 87016, 72183}, {16777216, 640, 189999, 166454, 103317},
         {16777216, 640, 50000, 54000, 54804}, {16777216, 640, 100000, 112056, 69529}, {16777216, 640, 189999, 219279, 96622},
         {4194304, 1400, 50000, 10403, 19810}, {4194304, 1400, 100000, 20757, 23886}, {4194304, 1400, 279999, 58478, 38712},
         {16777216, 128, 50000, 27578, 40600}, {16777216, 128, 100000, 52991, 56794}, {16777216, 128, 129999, 67933, 65335}};
    int bad = 0;
    for (const auto &r : t) {
        const uint64_t words = (((uint64_t)r[0] + 63) / 64 + 1) & ~1ull;
        const bool stream = sg::support_streams((uint64_t)r[2], (uint32_t)r[1], words);
        const double got = stream ? r[3] : r[4], other = stream ? r[4] : r[3];
        if (got > 1.1 * other) {
            std::printf("%.0f x %.0f, %.0f candidates: %s\n", r[0], r[1], r[2], stream ? "streamed" : "staged");
            ++bad;
        }
    }
    // the smallest and the largest calls
    if (!sg::support_streams(1, 1, 2) || !sg::support_streams(200, 40, 314)) return 2;
    if (sg::support_streams(1000000, 1024, 16384) || sg::support_streams(1ull << 32, 1792, 1ull << 20)) return 3;
    std::printf("%s\n", bad ? "slower" : "ok");
    return bad != 0;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_support_line_takes_the_faster_side(tmp_path):
    src, exe = tmp_path / "rule.cpp", tmp_path / "rule"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-O2", "-std=c++17", f"-I{CSRC}", str(src), "-o", str(exe)], check=True, timeout=120)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and r.stdout.strip().endswith("ok"), r.stdout + r.stderr
