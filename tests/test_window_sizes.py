"""The batched window miner's workspace sizes (csrc/window_sizes.h) on the CPU: the vertical rows hold every
window that its lists accept, and the word offsets of the 128 rows fit the 32 bits the kernel counts them in,
up to the longest window an API call takes (2^32 - 1 transactions)."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "20261008-self-growing-evidence-agent_gb300", "csrc")

PROGRAM = r"""
#include <cstdio>
#include "window_sizes.h"

int main() {
    const uint64_t lens[] = {0, 1, 31, 32, 33, 511, 65536, 65537, (1ull << 30) - 1024, (1ull << 30) - 1, 1ull << 30,
                             (1ull << 30) + 1, (1ull << 30) + (1ull << 24), 1ull << 31, (1ull << 32) - 1};
    for (uint64_t n : lens) {
        const sg::WindowSizes s = sg::window_sizes(n, true);
        const uint64_t fits = n < s.list_cap ? n : s.list_cap;   // entries of the largest task that is not refused
        const uint64_t words = ((fits + 31) / 32 + 3) & ~3ull;
        if (s.v_words < words || (s.v_words & 3)) { std::printf("%llu: rows of %llu words\n", (unsigned long long)n, (unsigned long long)s.v_words); return 1; }
        if (127 * s.v_words + words > 1ull << 32) { std::printf("%llu: offsets past 32 bits\n", (unsigned long long)n); return 1; }
        if (sg::window_sizes(n, false).v_words) return 1;
    }
    std::printf("ok\n");
    return 0;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_window_row_offsets_fit_32_bits(tmp_path):
    src, exe = tmp_path / "sizes.cpp", tmp_path / "sizes"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-O2", "-std=c++17", f"-I{CSRC}", str(src), "-o", str(exe)], check=True, timeout=120)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and r.stdout.strip().endswith("ok"), r.stdout + r.stderr
