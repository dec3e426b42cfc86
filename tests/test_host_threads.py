"""The helper threads of the host conversions (implexity_b200/csrc/lbm_host.h)
when memory for another one is not to be had."""
import shutil
import subprocess
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "implexity_b200" / "csrc"

PROGRAM = r"""
#include <cstdio>
#include <cstdlib>
#include <new>
#include <vector>

#include "lbm_host.h"

static thread_local int countdown = -1;  // allocations of this thread until one fails
void* operator new(std::size_t n) {
    if (countdown > 0 && --countdown == 0) throw std::bad_alloc();
    if (void* p = std::malloc(n)) return p;
    throw std::bad_alloc();
}
void operator delete(void* p) noexcept { std::free(p); }
void operator delete(void* p, std::size_t) noexcept { std::free(p); }

int main() {
    const int64_t n = (64 << 16) + 5;
    std::vector<unsigned char> seen((size_t)n);
    for (int fail = 0; fail < 40; ++fail) {
        std::fill(seen.begin(), seen.end(), 0);
        bool threw = false;
        countdown = fail > 0 ? fail : -1;
        try {
            lbm::parallel_range(n, [&](int64_t b, int64_t e) {
                for (int64_t i = b; i < e; ++i) ++seen[(size_t)i];
            });
        } catch (const std::bad_alloc&) {
            threw = true;
        }
        countdown = -1;
        // the first allocation is the shared job's, before any helper runs
        if (threw && fail != 1) return std::printf("threw at allocation %d\n", fail), 1;
        for (int64_t i = 0; i < n && !threw; ++i)
            if (seen[(size_t)i] != 1) return std::printf("value %lld done %d times at %d\n", (long long)i, seen[(size_t)i], fail), 1;
    }
    return 0;
}
"""


def test_no_exception_leaves_while_helpers_run(tmp_path):
    cxx = "/usr/bin/g++" if Path("/usr/bin/g++").exists() else shutil.which("g++")
    src, exe = tmp_path / "helpers.cpp", tmp_path / "helpers"
    src.write_text(PROGRAM)
    subprocess.run([cxx, "-std=c++17", "-O1", "-pthread", "-I", str(CSRC), str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, (r.returncode, r.stdout, r.stderr)
