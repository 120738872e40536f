"""The run-time divider of the transform kernels (csrc/fast_div.cuh), compiled for the
host: every divisor the kernels can see, up to the largest quotients they form."""
import os
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "channel-dns_b200", "csrc")
PROGRAM = """
#define __host__
#define __device__
#define __forceinline__ inline
#include "fast_div.cuh"
#include <cstdio>
int main() {
    for (int d = 1; d <= 700; ++d) {
        const cdns::FastDiv by(d);
        for (long long x = 0; x * d < (1LL << 32) && x < 20000; ++x)
            if (by((int)x) != x / d) return std::printf("%lld / %d -> %d\\n", x, d, by((int)x)), 1;
        const long long top = ((1LL << 32) - 1) / d;
        for (long long x = top > 0x7fffffff ? 0x7fffffff : top, k = 0; k < 2000; --x, ++k)
            if (by((int)x) != x / d) return std::printf("%lld / %d -> %d\\n", x, d, by((int)x)), 1;
    }
    return 0;
}
"""


def test_divider(tmp_path):
    src, exe = tmp_path / "div.cpp", tmp_path / "div"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-O2", "-std=c++17", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
