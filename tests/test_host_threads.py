"""Work split over host threads: every element once, also where threads cannot
be started (a process without room for their stacks), and no exception."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SRC = r"""
#include "sw2d_threads.h"
#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <sys/resource.h>
#include <unistd.h>

int main(int argc, char** argv) {
    const size_t n = std::strtoul(argv[1], nullptr, 10), nt = std::strtoul(argv[2], nullptr, 10);
    const long room = std::atol(argv[3]); /* megabytes left to the process (0: no limit) */
    std::vector<std::atomic<int>> seen(n);
    std::atomic<int> calls(0);
    if (room > 0) {
        std::FILE* f = std::fopen("/proc/self/statm", "r");
        unsigned long pages = 0;
        if (!f || std::fscanf(f, "%lu", &pages) != 1) return 3;
        std::fclose(f);
        rlimit r;
        r.rlim_cur = r.rlim_max = pages * (rlim_t)sysconf(_SC_PAGESIZE) + ((rlim_t)room << 20);
        if (setrlimit(RLIMIT_AS, &r) != 0) return 3;
    }
    sw2d::split_over_threads(n, nt, [&](size_t a, size_t b) {
        calls++;
        if (a >= b || b > n) std::abort();
        for (size_t k = a; k < b; k++) seen[k]++;
    });
    for (auto& s : seen)
        if (s != 1) return 4;
    std::printf("%d\n", calls.load());
    return 0;
}
"""


@pytest.fixture(scope="module")
def exe(tmp_path_factory):
    d = tmp_path_factory.mktemp("th")
    (d / "t.cpp").write_text(SRC)
    subprocess.check_call(["g++", "-std=c++17", "-O2", "-Wall", "-pthread", "-I",
                           os.path.join(ROOT, "sw2d_efdc_gb300", "csrc"), str(d / "t.cpp"), "-o", str(d / "t")])
    return str(d / "t")


@pytest.mark.parametrize("n,nt", [(1, 0), (1, 1), (1, 16), (7, 16), (16, 16), (17, 16), (100_000, 0), (100_000, 1),
                                  (100_000, 3), (100_000, 16)])
@pytest.mark.parametrize("room", [0, 1, 20])
def test_every_element_once(exe, n, nt, room):
    r = subprocess.run([exe, str(n), str(nt), str(room)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, (r.returncode, r.stderr)
    per = -(-n // nt) if nt > 1 else n
    pieces = -(-n // per)
    calls = int(r.stdout)
    assert calls == pieces if room == 0 else calls <= pieces
    if room == 1 and pieces > 1:  # no stack fits: the caller did it all
        assert calls == 1
