"""The set-up code's host-thread loop where the system starts no more threads (an
address-space limit that leaves no room for their stacks): every index is still
visited once, and no exception leaves the loop."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include <sys/resource.h>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include "host_parallel.h"

int main(int argc, char **argv) {
    static int seen[100000];
    if (argc > 1) {
        long kb = 0;
        char line[256];
        std::FILE *f = std::fopen("/proc/self/status", "r");
        while (std::fgets(line, sizeof line, f))
            if (!std::strncmp(line, "VmSize:", 7)) kb = std::atol(line + 7);
        std::fclose(f);
        rlimit r{};
        r.rlim_cur = r.rlim_max = (rlim_t)(kb + 1024) * 1024;   // a thread's stack takes 8 MiB
        if (setrlimit(RLIMIT_AS, &r)) return 3;
    }
    bsg::parallel_for(100000, 10, [&](int64_t i) { ++seen[i]; }, 32);
    for (int x : seen)
        if (x != 1) return 2;
    std::puts("ok");
    return 0;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_loop_without_room_for_threads(tmp_path):
    src, exe = tmp_path / "loop.cpp", tmp_path / "loop"
    src.write_text(PROGRAM)
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-pthread", "-I" + os.path.join(ROOT, "bigstickpublick_b200", "csrc"),
                           str(src), "-o", str(exe)])
    for args in ([], ["limit"]):
        r = subprocess.run([str(exe)] + args, capture_output=True, text=True)
        assert r.returncode == 0 and r.stdout == "ok\n", (args, r.returncode, r.stderr)
