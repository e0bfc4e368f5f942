"""The cut of the fp4 co-occurrence product (csrc/cooc_plan.h) on the CPU: over row counts on both sides of its
tiles and word counts on both sides of its steps, every tile meets every step exactly once, no accumulator
takes more steps than stay exact, and no CTA's work (its steps, and 7.5 of them for every unit whose counts it
adds to the output) is far above an even share of both."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "20261008-self-growing-evidence-agent_gb300", "csrc")

PROGRAM = r"""
#include <cstdio>
#include <vector>
#include "cooc_plan.h"

static int check(uint32_t d, uint64_t words, uint64_t n_sm) {
    const sg::F4Work w = sg::f4_plan(d, words, n_sm);
    const uint64_t steps = (words + 7) / 8;
    const uint32_t rows = (d + 127) / 128, cols = (d + 255) / 256;
    std::vector<std::vector<uint8_t>> seen(rows * cols);
    uint64_t found = 0;
    double most = 0;
    for (uint64_t c = 0; c < w.ctas; ++c) {
        uint64_t g, g1;
        double cost = 0;
        sg::f4_part(w, c, g, g1);
        if (g >= g1) { std::printf("%u x %llu: CTA %llu has nothing\n", d, (unsigned long long)words, (unsigned long long)c); return 1; }
        while (g < g1) {
            uint32_t bi, bj;
            uint64_t step0;
            const uint64_t follow = sg::f4_unit(w, g, bi, bj, step0), n = follow < g1 - g ? follow : g1 - g;
            if (bi >= rows || bj >= cols || bj < bi / 2 || n == 0 || step0 + n > steps || n > sg::kF4MaxSteps) {
                std::printf("%u x %llu: bad unit\n", d, (unsigned long long)words);
                return 1;
            }
            auto &s = seen[bi * cols + bj];
            s.resize(steps);
            for (uint64_t k = step0; k < step0 + n; ++k) if (s[k]++) { std::printf("%u x %llu: twice\n", d, (unsigned long long)words); return 1; }
            found += n;
            cost += n + 7.5;
            g += n;
        }
        if (cost > most) most = cost;
    }
    if (found != w.tiles * steps) { std::printf("%u x %llu: %llu of %llu steps\n", d, (unsigned long long)words, (unsigned long long)found, (unsigned long long)(w.tiles * steps)); return 1; }
    // an even share of the steps and of the tiles, a quarter more, and two units more for what does not divide evenly
    const uint64_t even = (w.total + n_sm - 1) / n_sm;
    const double least = even + 7.5 * ((w.tiles + n_sm - 1) / n_sm);
    if (most > 1.25 * least + 15.0) { std::printf("%u x %llu: a CTA's work %.1f, an even share %.1f\n", d, (unsigned long long)words, most, least); return 1; }
    return 0;
}

int main() {
    const uint32_t ds[] = {1, 64, 126, 128, 129, 256, 257, 300, 512, 640, 700, 900, 1024, 1051, 1238, 1400, 1792, 2500, 5000, 9000};
    const uint64_t ws[] = {2, 8, 10, 16, 24, 78, 128, 130, 256, 512, 514, 608, 688, 966, 1006, 1026, 1324, 2048, 3000, 4098, 8194, 16384, 16386, 40000};
    for (uint32_t d : ds)
        for (uint64_t w : ws)
            if ((uint64_t)d * w < 40000000 && (check(d, w, 152) || check(d, w, 148))) return 1;
    std::printf("ok\n");
    return 0;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_cooc_work_is_dealt_once_and_evenly(tmp_path):
    src, exe = tmp_path / "plan.cpp", tmp_path / "plan"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-O2", "-std=c++17", f"-I{CSRC}", str(src), "-o", str(exe)], check=True, timeout=120)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip().endswith("ok"), r.stdout + r.stderr
