"""The host threads that move a container's slices out of the staging ring: every size, with as many threads as the system
grants, and no thread left behind when a copy fails or a thread cannot be started."""
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "ptwm_b200", "csrc")
PROGRAM = r"""
#include "slice_copy.hpp"
#include <cstdio>
#include <cstdlib>
using namespace ptwm;
int main(int argc, char** argv) {
    const size_t n = std::atoll(argv[1]), slice = 64, ring = 3;
    const int granted = std::atoi(argv[2]);
    const long bad_send = std::atol(argv[3]), bad_arrival = std::atol(argv[4]);
    std::vector<uint8_t> src(n), dst(n, 0), stage(slice * ring);
    for (size_t i = 0; i < n; ++i) src[i] = uint8_t(i * 31 + i / 251);
    int started = 0;
    size_t sends = 0;
    auto start = [&](auto& f) {
        if (started >= granted) throw std::system_error(std::make_error_code(std::errc::resource_unavailable_try_again));
        ++started;
        return std::thread(f);
    };
    const Moved m = move_slices(dst.data(), stage.data(), n, slice, ring, 4,
        [&](size_t k) { ++sends; std::memcpy(stage.data() + k % ring * slice, src.data() + k * slice, std::min(slice, n - k * slice)); return long(k) != bad_send; },
        [&](size_t k) { return long(k) != bad_arrival; }, start);
    std::printf("%s %d %d", m == Moved::all ? "all" : m == Moved::failed ? "failed" : "no_threads", int(src == dst), int(sends > 0));
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("slice_copy")
    (d / "t.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-I", CSRC, "-o", str(d / "t"), str(d / "t.cpp")], check=True)
    return lambda *args: subprocess.run([str(d / "t"), *map(str, args)], check=True, capture_output=True, text=True, timeout=60).stdout.split()


@pytest.mark.parametrize("threads", [1, 2, 4])
@pytest.mark.parametrize("n", [1, 64, 65, 64 * 3, 64 * 3 + 1, 64 * 200 + 7])
def test_moves_every_slice(program, n, threads):
    assert program(n, threads, -1, -1) == ["all", "1", "1"]


def test_no_thread_can_be_started(program):
    assert program(64 * 20, 0, -1, -1) == ["no_threads", "0", "0"]  # nothing sent: the caller copies in another way


@pytest.mark.parametrize("threads", [1, 4])
@pytest.mark.parametrize("send,arrival", [(0, -1), (7, -1), (19, -1), (-1, 0), (-1, 7), (-1, 19)])
def test_a_failed_copy_ends_the_call(program, threads, send, arrival):
    assert program(64 * 20, threads, send, arrival)[0] == "failed"
