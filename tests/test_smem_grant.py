"""The shared-memory limit of a kernel that several threads launch with different sizes (csrc/tq_grant.h): it never goes down, and
what is noted as granted is what was set last.  Host code, compiled here against a stand-in for the runtime's call."""
import os
import shutil
import subprocess

import pytest

_MAIN = r"""
#include "tq_grant.h"
#include <chrono>
#include <cstdio>
#include <thread>
#include <vector>
int main() {
    for (int round = 0; round < 20; ++round) {
        TqSmemGrant grant;
        std::atomic<int> limit{0}, calls{0};
        std::atomic<bool> bad{false};
        std::vector<std::thread> threads;
        for (int size : {100, 200, 150, 50, 200, 120})
            threads.emplace_back([&, size] {
                const int error = grant.raise(3, size, [&](int want) {
                    // the smaller, the slower: a small limit that is set behind a large one would stand
                    std::this_thread::sleep_for(std::chrono::milliseconds((250 - want) / 25));
                    if (want < limit.load()) bad = true;
                    limit = want;
                    ++calls;
                    return 0;
                });
                if (error != 0 || limit.load() < size) bad = true;      // this thread's launch would be refused
            });
        for (auto& t : threads) t.join();
        if (bad || limit != 200 || grant.granted[3] != 200) { std::printf("limit %d, noted %d\n", limit.load(), grant.granted[3].load()); return 1; }
        const int before = calls;
        grant.raise(3, 200, [&](int) { ++calls; return 0; });            // granted already
        if (calls != before) return 2;
        if (grant.raise(5, 10, [](int) { return 7; }) != 7 || grant.granted[5] != 0) return 3;     // an error is handed on, and not noted
    }
    return 0;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs a host compiler")
def test_limit_only_grows(tmp_path):
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    source, program = tmp_path / "main.cpp", tmp_path / "main"
    source.write_text(_MAIN)
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-I", os.path.join(root, "project_tensor_b200", "csrc"), str(source), "-o", str(program)], check=True)
    done = subprocess.run([str(program)], capture_output=True, text=True, timeout=120)
    assert done.returncode == 0, (done.returncode, done.stdout)
