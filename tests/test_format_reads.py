"""The chunk classifier on the few bytes the plane entry points fetch of a payload: it looks at nothing behind them."""
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "ptwm_b200", "csrc")
PROGRAM = r"""
#define __host__
#define __device__
#include "format.hpp"
#include <cstdio>
#include <cstdlib>
#include <memory>
int main() {
    const uint16_t codec = std::atoi(argv[1]);
    std::unique_ptr<uint8_t[]> head(new uint8_t[6]{1, 100, 0, 0, 0, 40});  // tag, length, first byte of the coded bytes
    ptwm::ChunkDesc ch{};
    ch.body_len = 400; ch.decoded = 100;
    ptwm::detail::classify_chunk(head.get(), codec, ch);
    std::printf("%d %d %d", int(ch.raw), int(ch.data_off), int(ch.data_len));
}
"""


@pytest.mark.parametrize("codec", ["C_HUFFMAN", "C_RANS", "C_TANS"])
def test_classifier_reads_the_head_alone(tmp_path, codec):
    (tmp_path / "t.cpp").write_text(PROGRAM.replace("std::atoi(argv[1])", "ptwm::" + codec))
    subprocess.run(["g++", "-std=c++17", "-g", "-fsanitize=address", "-pthread", "-I", CSRC, "-o", str(tmp_path / "t"), str(tmp_path / "t.cpp")], check=True)
    run = subprocess.run([str(tmp_path / "t")], capture_output=True, text=True)
    assert run.returncode == 0, run.stderr[-2000:]
    assert run.stdout.split() == ["0", "5", "395"]
