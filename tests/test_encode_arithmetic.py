"""Host arithmetic the encoder's kernels share, over the whole range of plane lengths."""
import os
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "ptwm_b200", "csrc")
PROGRAM = r"""
#define __host__
#define __device__
#include "encode_tables.cuh"
#include <cstdio>
int main() {
    unsigned long long n;
    while (std::scanf("%llu", &n) == 1) std::printf("%u\n", ptwm::tans_encode_run(uint32_t(n)));
}
"""


def test_tans_runs_cover_every_length(tmp_path):
    (tmp_path / "t.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-I", CSRC, "-o", str(tmp_path / "t"), str(tmp_path / "t.cpp")], check=True)
    lengths = [1, 31, 32, 256, 8191, 8192, 8193, 8224, 65536, 2**31 - 1, 2**31, *range(2**32 - 70, 2**32)]
    out = subprocess.run([str(tmp_path / "t")], input="\n".join(map(str, lengths)), check=True, capture_output=True, text=True).stdout
    for n, run in zip(lengths, map(int, out.split()), strict=True):
        assert (n - 1) // run < 32, n  # 32 lanes are enough
        assert run == max(256, -(-n // 32)), n
