"""Host work on threads when memory or threads run out: every allocation that
starting them makes fails in turn, and the work is done by those there are."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

DRIVER = r"""
#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <new>
#include "host_threads.h"
static std::atomic<int> left{-1};  // allocations until they fail (-1: never)
void* operator new(std::size_t n)
{
    const int l = left.load();
    if (l == 0) throw std::bad_alloc();
    if (l > 0) left = l - 1;
    if (void* p = std::malloc(n)) return p;
    throw std::bad_alloc();
}
void operator delete(void* p) noexcept { std::free(p); }
void operator delete(void* p, std::size_t) noexcept { std::free(p); }
int main()
{
    for (int fail = 0; fail < 20; ++fail)
        for (unsigned threads : {0u, 1u, 2u, 16u}) {
            std::atomic<int> next{0}, done{0};
            left = fail;
            omv::on_threads(threads, [&] {
                while (next.fetch_add(1) < 1000) ++done;
            });
            left = -1;
            if (done != 1000) return 1;
        }
    std::puts("ok");
}
"""


def test_threads_that_cannot_be_started_are_left_out(tmp_path):
    (tmp_path / "driver.cpp").write_text(DRIVER)
    csrc = os.path.join(ROOT, "openmaterial-validation_gb300", "csrc")
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-I", csrc, str(tmp_path / "driver.cpp"), "-o",
                    str(tmp_path / "driver")], check=True)
    r = subprocess.run([str(tmp_path / "driver")], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and r.stdout == "ok\n", r
