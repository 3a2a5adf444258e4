"""The shared-memory opt-in of a kernel (csrc/shared_limit.h) from several threads.

The limit is the process's; a handle set up for a larger mesh relies on it for
good.  The fake limit's reader is slow for the smaller request, so that
without a lock its write lands last.
"""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include <atomic>
#include <chrono>
#include <cstdio>
#include <stdexcept>
#include <thread>

#include "shared_limit.h"

static std::atomic<std::size_t> limit{48};

static void ask(std::size_t want, int ms) {
    fea::raise_shared_limit(
        want,
        [&] {
            const std::size_t now = limit;
            std::this_thread::sleep_for(std::chrono::milliseconds(ms));
            return now;
        },
        [](std::size_t n) { limit = n; });
}

int main() {
    std::thread small(ask, 60, 300), large(ask, 100, 50);
    small.join();
    large.join();
    const std::size_t both = limit;
    ask(80, 0);  // never lowered
    try {        // a failing call leaves no lock behind
        fea::raise_shared_limit(500, []() -> std::size_t { throw std::runtime_error("no"); }, [](std::size_t) {});
    } catch (const std::runtime_error&) {
    }
    std::thread later(ask, 120, 0);
    later.join();
    std::printf("%zu %zu\n", both, limit.load());
}
"""


def test_the_larger_request_stays(tmp_path):
    src, exe = tmp_path / "limit.cpp", tmp_path / "limit"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-pthread", "-I", os.path.join(ROOT, "fea-visualizer_gb300", "csrc"), str(src),
                    "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True, timeout=60).stdout
    assert out.split() == ["100", "120"]
