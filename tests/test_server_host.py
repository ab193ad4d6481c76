"""The request server's host side, without a GPU: its source is compiled into a
small program in which the CUDA calls it makes are recorded."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "string-sorting_b200")
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")

PRELUDE = r"""
#include <cuda.h>
#include <cuda_runtime.h>
#include <cstdint>
#include <cstdio>
#include <string>
#include <vector>

static std::vector<std::string> calls;  // what the server asked of the device
static int failed = 0;
#define CHECK(x) \
    if (!(x)) std::printf("line %d: %s\n", __LINE__, #x), failed = 1

// Pointers below 1 << 20 stand for memory of device 0.
static bool is_device(const void *p) { return (uintptr_t)p < (1 << 20); }
static cudaError_t fake_attributes(cudaPointerAttributes *at, const void *p) {
    calls.push_back("attributes");
    *at = cudaPointerAttributes{};
    at->type = is_device(p) ? cudaMemoryTypeDevice : cudaMemoryTypeHost;
    return cudaSuccess;
}
static cudaError_t fake_copy(void *, const void *, size_t n, cudaMemcpyKind, cudaStream_t) {
    calls.push_back("copy " + std::to_string(n));
    return cudaSuccess;
}
static cudaError_t fake_set(void *, int, size_t n, cudaStream_t) {
    calls.push_back("set " + std::to_string(n));
    return cudaSuccess;
}
static cudaError_t fake_record(cudaEvent_t e, cudaStream_t) {
    calls.push_back("record " + std::to_string((uintptr_t)e));
    return cudaSuccess;
}
static cudaError_t fake_create(cudaEvent_t *e, unsigned) {
    static uintptr_t made = 0;
    *e = (cudaEvent_t)++made;
    return cudaSuccess;
}
static cudaError_t fake_sync(cudaEvent_t) { return cudaSuccess; }
static cudaError_t fake_last() { return cudaSuccess; }
// Their allocations: 100 bytes at every multiple of 4096.
static CUresult fake_range(CUdeviceptr *base, size_t *size, CUdeviceptr p) {
    *base = p & ~4095ull;
    *size = 100;
    return p - *base < 100 ? CUDA_SUCCESS : CUDA_ERROR_NOT_FOUND;
}
static cudaError_t fake_entry(const char *name, void **f, unsigned, unsigned long long,
                              cudaDriverEntryPointQueryResult *q) {
    CHECK(std::string(name) == "cuMemGetAddressRange");
    *f = (void *)fake_range;
    *q = cudaDriverEntryPointSuccess;
    return cudaSuccess;
}
#define cudaGetDriverEntryPointByVersion fake_entry
#define cudaPointerGetAttributes fake_attributes
#define cudaMemcpyAsync fake_copy
#define cudaMemsetAsync fake_set
#define cudaEventRecord fake_record
#define cudaEventCreateWithFlags fake_create
#define cudaEventSynchronize fake_sync
#define cudaGetLastError fake_last
#include "ssort_server.cu"

namespace ssort {
void launch_copies(const CopyJob *, uint32_t njobs, uint32_t, cudaStream_t) {
    calls.push_back("copies " + std::to_string(njobs));
}
}  // namespace ssort

template <class T = uint8_t>
static T *at(uintptr_t p) { return (T *)p; }

// A server of 1 MB and `strings` positions that has seen no device.
struct Made {
    ssort_ctx ctx;
    ssort_server srv;
    std::vector<CopyJob> jobs[2];
    explicit Made(uint32_t strings = 100000) {
        srv.ctx = &ctx;
        srv.budget = 1 << 20;
        srv.max_strings = strings;
        srv.arena_alloc.init(srv.budget);
        srv.pos_alloc.init(strings);
        ctx.num_sms = 148;
        for (int k = 0; k < 2; ++k) {
            jobs[k].resize(CopyBatch::CAP);
            (k ? srv.out : srv.in).h = jobs[k].data();
        }
    }
    uint64_t submit(const uint8_t *arena, uint64_t bytes, const void *offs, uint64_t n,
                    uint32_t *perm, uint32_t *lcp = nullptr) {
        uint64_t id = 0;
        CHECK(ssort_server_submit(&srv, arena, bytes, offs, 8, n, perm, lcp, &id) == SSORT_OK);
        return id;
    }
};
static std::string joined() {
    std::string s;
    for (auto &c : calls) s += c + ", ";
    return s;
}
"""


def run(tmp_path, body):
    if not os.path.exists(os.path.join(CUDA, "lib64", "libcudart_static.a")):
        pytest.skip("no CUDA toolkit")
    src = tmp_path / "server.cpp"
    src.write_text(PRELUDE + "int main() {\n" + body + "\n    return failed;\n}\n")
    exe = tmp_path / "server"
    subprocess.run(["/usr/bin/g++", "-std=c++17", "-w", "-I", os.path.join(CUDA, "include"),
                    "-I", os.path.join(ROOT, "include"), "-I", os.path.join(PKG, "csrc"),
                    str(src), "-o", str(exe), os.path.join(PKG, "libssort_b200.so"),
                    "-Wl,-rpath," + PKG, "-L", os.path.join(CUDA, "lib64"), "-lcudart_static",
                    "-ldl", "-lrt", "-lpthread"], check=True)
    r = subprocess.run([str(exe)], stdout=subprocess.PIPE, text=True, timeout=60)
    assert r.returncode == 0, r.stdout


def test_submit_asks_nothing_of_the_device(tmp_path):
    """A submit from a thread that has made no CUDA call must not bring up a
    context on whichever device is current there: where the buffers lie is found
    out when the request is admitted, on the server's device."""
    run(tmp_path, r"""
    Made m;
    m.submit(at(0x1000), 100, at(0x2000), 5, at<uint32_t>(0x3000), at<uint32_t>(0x4000));
    m.submit(at(1ull << 40), 100, at(2ull << 40), 5, at<uint32_t>(3ull << 40));
    CHECK(calls.empty());
    CHECK(m.srv.admit() == SSORT_OK);
    CHECK(m.srv.loading.size() == 2);
    CHECK(m.srv.loading[0]->dev_in && m.srv.loading[0]->dev_out);
    CHECK(!m.srv.loading[1]->dev_in && !m.srv.loading[1]->dev_out);
    """)


def test_copies_beyond_an_allocation_go_through_the_driver(tmp_path):
    """cudaMemcpyAsync refuses a range that leaves its allocation; a kernel that
    copies does not.  Only buffers that lie inside their allocations in full are
    copied by the server's kernel, inputs and outputs apart."""
    run(tmp_path, r"""
    // allocations of 100 bytes at every multiple of 4096
    {
        Made m;
        // n = 10: 80 bytes of offsets, 40 of results
        m.submit(at(0x1000), 100, at(0x2000 + 20), 10, at<uint32_t>(0x3000 + 60),
                 at<uint32_t>(0x4000));
        CHECK(m.srv.admit() == SSORT_OK);
        CHECK(m.srv.loading[0]->dev_in && m.srv.loading[0]->dev_out);
        CHECK(joined().find("copies 2") != std::string::npos);
    }
    struct { uintptr_t arena, bytes, offs, perm, lcp; bool in, out; } bad[] = {
        {0x1000, 101, 0x2000, 0x3000, 0x4000, false, true},
        {0x1000 + 1, 100, 0x2000, 0x3000, 0x4000, false, true},
        {0x1000, 100, 0x2000 + 21, 0x3000, 0x4000, false, true},
        {0x1000, 100, 0x2000, 0x3000 + 61, 0x4000, true, false},
        {0x1000, 100, 0x2000, 0x3000, 0x4000 + 61, true, false},
        {0x1000, ~0ull >> 45, 0x2000, 0x3000, 0x4000, false, true},
        {0x1000 + 200, 1, 0x2000, 0x3000, 0x4000, false, true},  // in none
    };
    for (auto &b : bad) {
        calls.clear();
        Made m;
        m.submit(at(b.arena), b.bytes, at(b.offs), 10, at<uint32_t>(b.perm),
                 at<uint32_t>(b.lcp));
        CHECK(m.srv.admit() == SSORT_OK);
        CHECK(m.srv.loading[0]->dev_in == b.in);
        CHECK(m.srv.loading[0]->dev_out == b.out);
        const bool plain = joined().find("copy " + std::to_string(b.bytes) + ",") !=
                           std::string::npos;
        CHECK(plain == !b.in);
        CHECK((joined().find("copies 2") != std::string::npos) == b.in);
    }
    """)


def test_a_host_request_waits_for_its_own_copies_only(tmp_path):
    """Requests admitted in one step: a host request's event follows its own
    copies and comes before the next one's; device requests next to each other
    share a launch, whose events come before the copies of a later host request."""
    run(tmp_path, r"""
    const uintptr_t H = 1ull << 40;
    Made m;
    // host, host, device, device, host, device; n = 1, 2, .. marks the offsets' copies
    for (int i = 1; i <= 6; ++i) {
        const bool dev = i == 3 || i == 4 || i == 6;
        const uintptr_t base = dev ? 0 : H;
        m.submit(at(base + 0x1000 * i), 10 * i, at(base + 0x10000), i,
                 at<uint32_t>(base + 0x20000));
    }
    CHECK(m.srv.admit() == SSORT_OK);
    CHECK(m.srv.loading.size() == 6);
    std::vector<std::string> seen;  // without the queries and the table's own copy and event
    for (auto &c : calls)
        if (c != "attributes" && c != "record 0" && c.compare(0, 3, "set") &&
            c != "copy " + std::to_string(4 * sizeof(CopyJob)) &&
            c != "copy " + std::to_string(2 * sizeof(CopyJob)))
            seen.push_back(c);
    const std::vector<std::string> want = {
        "copy 10", "copy 8", "record 1", "copy 20", "copy 16", "record 2",
        "copies 4", "record 3", "record 4",
        "copy 50", "copy 40", "record 5", "copies 2", "record 6"};
    CHECK(seen == want);
    if (seen != want) for (auto &c : seen) std::printf("%s, ", c.c_str());
    """)


def test_rules_by_size_go_by_the_requests_held(tmp_path):
    """A round's tile and leaf sizes and samples per splitter are those of a sort
    of as many strings as the active requests hold, whatever the server could
    hold; the count matrix, sized for the latter, has room for them."""
    run(tmp_path, r"""
    const uint32_t CAPS[] = {50000, 300000, 1u << 20, 16u << 20, 100u << 20};
    const uint32_t SIZES[] = {2049, 75776, 75777, 300000, 606208, 606209, 1u << 20,
                              LEAF_MIN_N - 1, LEAF_MIN_N, 16u << 20, 100u << 20};
    for (uint32_t cap : CAPS) {
        Made m(cap);
        const WsLayout lay = ws_layout(cap);
        for (uint32_t n : SIZES) {
            if (n > cap) continue;
            Request a, b;
            a.n = n / 3;
            b.n = n - n / 3;
            m.srv.active = {&a, &b};
            const SortArgs s = m.srv.args();
            CHECK(s.n == n);
            CHECK(s.tile == part_tile(n));
            CHECK(s.leaf_cap == (n >= LEAF_MIN_N ? LEAF_CAP : SMALL_CAP));
            // tiles: one more for the remainder of each large segment
            const uint64_t tiles = n / s.tile + n / (SMALL_CAP + 1) + 1;
            CHECK(tiles * NB_MAX < lay.cm_cap);
        }
        m.srv.active.clear();
    }
    """)
