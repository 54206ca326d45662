"""CPU test of the staged host copies (st_xfer.cu) on a stand-in for the CUDA runtime: bytes, which
contexts the copies touch, captures on other threads, what is pinned, failing calls."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

DRIVER = r"""
#include <cassert>
#include <cstdio>
#include <thread>
#include <vector>
#include "st_xfer.h"

namespace fake {
std::atomic<int> set_device{0}, host_allocs{0}, copies{0}, syncs{0}, fail_copy{0};
std::atomic<long> host_bytes{0};
thread_local void* context = nullptr;
thread_local int mode = cudaStreamCaptureModeGlobal;
int primary_word, other_word;
void *primary = &primary_word, *stream_context = &primary_word;
bool refuse_alloc = false;
int global_capture = 0;
std::mutex mu;
std::set<void*> pinned;
}  // namespace fake
using namespace st;

static const size_t MB = (size_t)1 << 20;

/* Both directions of `bytes` bytes in three segments of odd sizes; whether all arrived. */
static bool both(size_t bytes, cudaError_t* err = nullptr)
{
    std::vector<unsigned char> a(bytes), dev(bytes, 0), b(bytes, 0);
    for (size_t i = 0; i < bytes; ++i) a[i] = (unsigned char)(i * 2654435761u >> 13);
    const size_t c1 = bytes / 3 | 1, c2 = bytes / 2 | 1;
    auto seg = [&](unsigned char* h, XferSeg* s) {
        s[0] = {h, dev.data(), c1};
        s[1] = {h + c1, dev.data() + c1, c2 - c1};
        s[2] = {h + c2, dev.data() + c2, bytes - c2};
    };
    XferSeg s[3];
    int stream = 0;
    seg(a.data(), s);
    cudaError_t e = xfer_up(s, 3, 0, &stream);
    seg(b.data(), s);
    if (e == cudaSuccess) e = xfer_down(s, 3, 0, &stream);
    if (err) *err = e;
    return e == cudaSuccess && a == b && a == dev;
}

int main(int argc, char** argv)
{
    const std::string what = argv[1];
    fake::context = fake::primary;
    xfer_retain();
    if (what != "on_demand" && what != "no_primary" && what != "own_context")
        assert(both(140 * MB));             /* copies are staged from now on */
    if (what == "bytes") {
        for (size_t n : {(size_t)9, 140 * MB, 2 * MB - 1, 2 * MB, 3 * MB + 5, 16 * MB - 7, 40 * MB + 3, 100 * MB + 1})
            assert(both(n));
        std::thread t([] {
            fake::context = fake::primary;
            for (int k = 0; k < 20; ++k) assert(both(7 * MB + k));
        });
        for (int k = 0; k < 20; ++k) assert(both(9 * MB + k));
        t.join();
    } else if (what == "own_context") {
        /* a handle in a context of the caller's: its copies arrive and its context stays */
        fake::context = fake::stream_context = &fake::other_word;
        assert(both(300 * MB));
        assert(fake::context == &fake::other_word && fake::set_device == 0);
        /* and one in the primary context afterwards */
        fake::context = fake::stream_context = fake::primary;
        assert(both(300 * MB));
        assert(fake::set_device > 0);
    } else if (what == "no_primary") {
        fake::primary = nullptr;
        fake::context = fake::stream_context = &fake::other_word;
        assert(both(300 * MB) && fake::context == &fake::other_word);
    } else if (what == "capture") {
        /* another thread captures in global mode, and the caller's may copy all the same */
        assert(both(100 * MB));
        fake::global_capture = 1;
        fake::mode = cudaStreamCaptureModeRelaxed;
        for (int k = 0; k < 5; ++k) assert(both(100 * MB));
        assert(fake::mode == cudaStreamCaptureModeRelaxed);
    } else if (what == "no_pinned") {
        xfer_release();
        xfer_retain();
        fake::refuse_alloc = true;
        assert(both(300 * MB));
    } else if (what == "on_demand") {
        /* nothing is pinned for small copies, or before 48 MB have been copied; then only what
         * the copy's threads use, at most 24 MB; and all of it goes with the last handle */
        for (int k = 0; k < 200; ++k) assert(both(2 * MB - 1));
        assert(fake::host_allocs == 0);
        for (int k = 0; k < 4; ++k) assert(both(5 * MB));
        assert(fake::host_allocs == 0);
        for (int k = 0; k < 5; ++k) assert(both(5 * MB));
        assert(fake::host_bytes > 0 && fake::host_bytes <= (long)(6 * MB));
        xfer_retain();
        for (int k = 0; k < 3; ++k) assert(both(100 * MB));
        assert(fake::pinned.size() == 1 && fake::host_bytes <= (long)(30 * MB));
        xfer_release();
        assert(!fake::pinned.empty());
        xfer_release();
        assert(fake::pinned.empty());
        const int n = fake::host_allocs;
        for (int k = 0; k < 5; ++k) {       /* one handle after another */
            xfer_retain();
            assert(both(20 * MB));
            xfer_release();
        }
        assert(fake::host_allocs == n);
        xfer_retain();                      /* a large transfer in chunks: from the first on */
        std::vector<unsigned char> a(30 * MB), dev(30 * MB);
        XferSeg s = {a.data(), dev.data(), 30 * MB};
        int stream = 0;
        assert(xfer_up(&s, 1, 0, &stream, 500 * MB) == cudaSuccess && fake::host_allocs == n + 1);
    } else if (what == "reset") {
        /* pinned pieces that are gone (a reset device) are not written to */
        assert(both(100 * MB));
        for (void* p : std::set<void*>(fake::pinned)) cudaFreeHost(p);
        assert(both(100 * MB));
    } else if (what == "failing_copy") {
        assert(both(100 * MB));
        for (int k = 1; k < 30; k += 4) {
            fake::copies = 0;
            fake::fail_copy = k;
            cudaError_t e;
            const int synced = fake::syncs;
            assert(!both(30 * MB, &e) && e == cudaErrorUnknown && fake::syncs > synced);
            fake::fail_copy = 0;
            assert(both(30 * MB));
        }
    } else {
        return 2;
    }
    xfer_release();
    assert(fake::pinned.empty());
    puts("ok");
    return 0;
}
"""


@pytest.fixture(scope="module")
def driver(tmp_path_factory):
    d = tmp_path_factory.mktemp("xfer")
    src = d / "driver.cpp"
    src.write_text("#include <string>\n" + DRIVER)
    exe = d / "driver"
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-pthread", "-I",
                           os.path.join(ROOT, "tests", "fake_cuda"), "-I",
                           os.path.join(ROOT, "scale-track_b200", "csrc"), str(src), "-x", "c++",
                           os.path.join(ROOT, "scale-track_b200", "csrc", "st_xfer.cu"), "-o",
                           str(exe)])
    return str(exe)


@pytest.mark.parametrize("what", ["bytes", "own_context", "no_primary", "capture", "no_pinned",
                                  "on_demand", "reset", "failing_copy"])
def test_staged_copies(driver, what):
    r = subprocess.run([driver, what], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout == "ok\n", r.stderr
