"""The counts that the host works with between two reads are its own: a kernel
that publishes its counters while the host launches the sorts of the level
before must not change them under it."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "string-sorting_b200")
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")

PROGRAM = r"""
#include <cstdio>
#include "ssort_host.cuh"
using namespace ssort;

static int failed = 0;
#define CHECK(x) \
    if (!(x)) std::printf("line %d: %s\n", __LINE__, #x), failed = 1

int main() {
    static HostCounters page{};  // stands for the pinned page that kernels write
    ssort_ctx c;
    c.hc = &page;
    c.published = true;
    c.use_counters(0);
    // a kernel publishes its counts; the host waits for them
    Publish p = c.publish_next();
    CHECK(p.host == (uint32_t *)&page);
    page.rc.c[0].n_w1 = 7;
    page.rc.c[1].n_next = 5;
    page.flag = p.seq;
    CHECK(c.read_counters() == SSORT_OK);
    CHECK(c.h_ctr->n_w1 == 7);
    // the next kernel publishes before the host has waited for it
    p = c.publish_next();
    page.rc.c[0].n_w1 = 99;
    page.rc.c[0].n_equal = 3;
    page.flag = p.seq;
    CHECK(c.h_ctr->n_w1 == 7);
    CHECK(c.h_ctr->n_equal == 0);
    c.use_counters(1);
    CHECK(c.h_ctr->n_next == 5);
    c.use_counters(0);
    CHECK(c.read_counters() == SSORT_OK);
    CHECK(c.h_ctr->n_w1 == 99);
    CHECK(c.h_ctr->n_equal == 3);
    // what the host writes stays out of the page, and an error is reported
    *c.h_ctr = Counters{};
    CHECK(page.rc.c[0].n_w1 == 99);
    p = c.publish_next();
    page.rc.c[1].error = 1;
    page.flag = p.seq;
    CHECK(c.read_counters() == SSORT_EINTERNAL);
    c.hc = nullptr;
    return failed;
}
"""


def test_counts_change_only_when_they_are_read(tmp_path):
    if not os.path.exists(os.path.join(CUDA, "include", "cuda_runtime.h")):
        pytest.skip("no CUDA headers")
    src = tmp_path / "counters.cpp"
    src.write_text(PROGRAM)
    exe = tmp_path / "counters"
    subprocess.run(["/usr/bin/g++", "-std=c++17", "-I", os.path.join(CUDA, "include"),
                    "-I", os.path.join(ROOT, "include"), "-I", os.path.join(PKG, "csrc"),
                    str(src), "-o", str(exe), os.path.join(PKG, "libssort_b200.so"),
                    "-Wl,-rpath," + PKG], check=True)
    r = subprocess.run([str(exe)], stdout=subprocess.PIPE, text=True, timeout=60)
    assert r.returncode == 0, r.stdout
