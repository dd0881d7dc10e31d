"""Populating the pages of result arrays, on the CPU: csrc/host_pages.cpp compiled with g++ against a madvise that
records the ranges it is given."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include <stdio.h>
#include <string.h>
#include <sys/mman.h>
#include <unistd.h>
#include <atomic>
#include "host_pages.h"
static std::atomic<long> calls{0}, bytes{0};
extern "C" int madvise(void *, size_t n, int) noexcept { ++calls; bytes += long(n); return 0; }
static void show(const char *what) { printf("%s %ld %ld\n", what, calls.load(), bytes.load()); calls = 0; bytes = 0; }
static char *fresh(size_t n) {
    return static_cast<char *>(mmap(nullptr, n, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0));
}
int main() {
    const size_t page = size_t(sysconf(_SC_PAGESIZE)), big = size_t(32) << 20, small = 8 * page;
    char *a = fresh(big), *b = fresh(small);
    fpt::populate_pages({{a, big}, {b, small}, {nullptr, big}, {a + 1, page}, {a, 0}});
    show("new");
    memset(a, 1, big);
    memset(b, 1, small);
    fpt::populate_pages({{a, big}, {b, small}});
    show("kept");
    char *c = fresh(big);
    memset(c, 1, big / 2);
    fpt::populate_pages({{c, big}});
    show("half");
    char *d = fresh(small);
    memset(d, 1, page);
    fpt::populate_pages({{d + 100, small - 200}});
    show("inner");
    printf("page %zu\n", page);
    return 0;
}
"""


@pytest.fixture(scope="module")
def recorded(tmp_path_factory):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("g++ is not available")
    tmp = tmp_path_factory.mktemp("pages")
    csrc = os.path.join(ROOT, "fractalpathtracer_gb300", "csrc")
    (tmp / "main.cpp").write_text(PROGRAM)
    exe = str(tmp / "pages")
    subprocess.run([gxx, "-std=c++17", "-Wall", "-I", csrc, str(tmp / "main.cpp"), os.path.join(csrc, "host_pages.cpp"),
                    "-o", exe, "-lpthread"], check=True, capture_output=True, text=True)
    out = subprocess.run([exe], check=True, capture_output=True, text=True).stdout
    return {line.split()[0]: [int(v) for v in line.split()[1:]] for line in out.splitlines()}


def test_new_arrays_are_populated_whole(recorded):
    page = recorded["page"][0]
    assert recorded["new"] == [5, (32 << 20) + 8 * page]      # four parts of the large array, one of the small
    assert recorded["half"] == [4, 32 << 20]
    assert recorded["inner"] == [1, 6 * page]                 # whole pages only


def test_kept_arrays_are_left_alone(recorded):
    assert recorded["kept"] == [0, 0]
