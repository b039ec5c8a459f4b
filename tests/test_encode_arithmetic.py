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
    while (std::scanf("%llu", &n) == 1)
        std::printf("%u %d %llu\n", ptwm::tans_encode_run(uint32_t(n)), int(ptwm::plane_codable(n)), (unsigned long long)ptwm::plane_slot_cap(n));
}
"""


def arithmetic(tmp_path, lengths):
    (tmp_path / "t.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-I", CSRC, "-o", str(tmp_path / "t"), str(tmp_path / "t.cpp")], check=True)
    out = subprocess.run([str(tmp_path / "t")], input="\n".join(map(str, lengths)), check=True, capture_output=True, text=True).stdout
    return [tuple(map(int, line.split())) for line in out.splitlines()]


def test_tans_runs_cover_every_length(tmp_path):
    lengths = [1, 31, 32, 256, 8191, 8192, 8193, 8224, 65536, 2**31 - 1, 2**31, *range(2**32 - 70, 2**32)]
    for n, (run, _, _) in zip(lengths, arithmetic(tmp_path, lengths), strict=True):
        assert (n - 1) // run < 32, n  # 32 lanes are enough
        assert run == max(256, -(-n // 32)), n


def test_single_planes_up_to_a_slot_of_a_gibibyte(tmp_path):
    longest = 4 * (((2**30 - 1 - 64) * 8) // 12 - 1) + 3  # twelve bits for a fourth of its symbols, and 64 bytes
    lengths = [1, 64, 200_000, *range(longest - 60, longest + 60)]
    for n, (_, codable, slot) in zip(lengths, arithmetic(tmp_path, lengths), strict=True):
        assert codable == (n <= longest), n
        assert slot % 16 == 0 and slot >= (n + 3) // 4 * 12 / 8 + 16, n
