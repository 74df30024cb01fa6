"""Host-side rules of the library (csrc/crt_host.h), compiled as plain C++ and
checked without a GPU."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def run_cpp(tmp_path, body):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("no g++")
    src, exe = tmp_path / "rule.cpp", tmp_path / "rule"
    src.write_text('''#include "crt_host.h"
#include <atomic>
#include <chrono>
#include <cstdio>
#include <cstdlib>
#include <thread>
#include <vector>
#define CHECK(c) do { if (!(c)) { std::printf("line %d: %s\\n", __LINE__, #c); return 1; } } while (0)
''' + body)
    subprocess.run([gxx, "-std=c++17", "-O1", "-pthread", "-Wall", "-Werror", "-I",
                    os.path.join(ROOT, "realtimeraytracing_gb300", "csrc"), str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout


def test_derived_data_is_enqueued_once_and_waited_for(tmp_path):
    """Contexts on threads of their own: one derives, every other one waits for a derivation that is already
    enqueued, the deriving one does neither again; a failed derivation is left to the next; a reset starts over."""
    run_cpp(tmp_path, r'''
enum Status { kOk = 0, kFailed = 3 };
int main() {
    for (int round = 0; round < 50; ++round) {
        crt::Derived d;
        std::atomic<int> derived{0}, waited{0}, early{0};
        std::atomic<bool> enqueued{false};
        std::vector<std::thread> t;
        for (uint64_t who = 1; who <= 8; ++who)
            t.emplace_back([&, who] {
                for (int k = 0; k < 3; ++k) {
                    bool did = false, saw = false;
                    const Status s = d.use(who,
                        [&] { ++derived; did = true; std::this_thread::sleep_for(std::chrono::microseconds(200));
                              enqueued = true; return kOk; },
                        [&] { ++waited; saw = true; if (!enqueued) ++early; return kOk; });
                    if (s != kOk || !enqueued || (did && saw)) ++early;
                }
            });
        for (auto& x : t) x.join();
        CHECK(derived == 1);
        CHECK(waited == 3 * 7);
        CHECK(early == 0);
        CHECK(d.ready());
    }
    crt::Derived d;
    int derived = 0, waited = 0;
    auto ok = [&] { ++derived; return kOk; };
    auto bad = [&] { ++derived; return kFailed; };
    auto wait = [&] { ++waited; return kFailed; };
    CHECK(d.use(1, bad, wait) == kFailed && derived == 1 && !d.ready());
    CHECK(d.use(2, ok, wait) == kOk && derived == 2 && d.ready());
    CHECK(d.use(2, ok, wait) == kOk && derived == 2 && waited == 0);
    CHECK(d.use(1, ok, wait) == kFailed && derived == 2 && waited == 1);  // the wait's own error
    d.reset();
    CHECK(!d.ready());
    CHECK(d.use(1, ok, wait) == kOk && derived == 3 && waited == 1);
    CHECK(d.use(2, ok, wait) == kFailed && waited == 2);
    return 0;
}
''')


def test_build_launches_fit_the_device_and_start_over_only_untouched(tmp_path):
    """Grids whose blocks wait for one another follow the device's SMs (152, or fewer), and a failure after the first
    launch is a failure: the launch-per-iteration path would read what that launch has overwritten."""
    run_cpp(tmp_path, r'''
int main() {
    for (int sms : {1, 76, 140, 152})
        for (int per_sm : {1, 2, 3, 8})
            for (int most : {2, 3, 64}) {
                const int g = crt::resident_blocks(true, per_sm, most, sms);
                CHECK(g > 0 && g % sms == 0 && g <= per_sm * sms && g <= most * sms);
                CHECK(g == per_sm * sms || g == most * sms);
            }
    CHECK(crt::resident_blocks(false, 3, 3, 152) == 0);
    CHECK(crt::resident_blocks(true, 0, 3, 152) == 0);
    CHECK(crt::resident_blocks(true, 3, 3, 0) == 0);
    CHECK((crt::PlocGrids{456, 304, 1216, 16}.supported()));
    CHECK((!crt::PlocGrids{0, 304, 1216, 16}.supported() && !crt::PlocGrids{456, 0, 1216, 16}.supported()));
    CHECK((!crt::PlocGrids{456, 304, 0, 16}.supported() && !crt::PlocGrids{456, 304, 1216, 0}.supported()));
    CHECK(crt::may_start_over(true, false));
    CHECK(!crt::may_start_over(true, true) && !crt::may_start_over(false, false) && !crt::may_start_over(false, true));
    return 0;
}
''')


def test_an_abandoned_calls_error_is_not_the_next_calls(tmp_path):
    """A call returns early while its kernels run; one of them raises an error afterwards.  The next call waits for
    them before it clears the words, and reports its own errors only."""
    run_cpp(tmp_path, r'''
enum Status { kOk = 0, kFailed = 3 };
int main() {
    uint32_t w[4] = {9, 9, 9, 9}, out[4];
    std::vector<uint32_t> queue;  // words that kernels in flight will raise
    int waits = 0;
    auto sync = [&] { ++waits; for (uint32_t e : queue) w[0] |= e; queue.clear(); return kOk; };
    auto dead = [&] { return kFailed; };
    crt::HostErrorWords e;
    e.words = w;
    CHECK(e.begin(sync) == kOk && waits == 0 && w[0] == 0 && w[3] == 0);
    CHECK(e.end(sync, out) == kOk && waits == 1 && out[0] == 0);
    CHECK(e.begin(sync) == kOk && waits == 1);  // nothing is in flight between calls: no wait
    queue.push_back(4);
    CHECK(e.end(sync, out) == kOk && out[0] == 4);
    CHECK(e.begin(sync) == kOk && waits == 2 && w[0] == 0);
    queue.push_back(16);  // and the call returns without end()
    CHECK(e.begin(sync) == kOk && waits == 3 && queue.empty() && w[0] == 0);
    queue.push_back(1);
    CHECK(e.end(sync, out) == kOk && out[0] == 1);
    CHECK(e.begin(sync) == kOk && e.end(dead, out) == kFailed);  // not known to be over: the next call waits
    CHECK(e.begin(dead) == kFailed);
    waits = 0;
    CHECK(e.begin(sync) == kOk && waits == 1);
    return 0;
}
''')


def test_scenes_and_cameras_the_compressed_walk_refuses(tmp_path):
    """The bounds, from both sides; what is not a number is refused."""
    run_cpp(tmp_path, r'''
#include <limits>
int main() {
    const float inf = std::numeric_limits<float>::infinity(), nan = std::nanf("");
    const float lo = std::ldexp(1.f, -60), hi = std::ldexp(1.f, 30);
    CHECK(crt::walk4_scene(lo) && crt::walk4_scene(hi) && crt::walk4_scene(1e-6f));
    CHECK(!crt::walk4_scene(std::nextafter(lo, 0.f)) && !crt::walk4_scene(std::nextafter(hi, inf)));
    CHECK(!crt::walk4_scene(inf) && !crt::walk4_scene(nan) && !crt::walk4_scene(0.f));
    const float eps = std::ldexp(3.f, -20);  // a scene of range 3
    for (int a = 0; a < 3; ++a)
        for (float sign : {1.f, -1.f}) {
            float e[3] = {0.5f, 0.5f, -1.5f};
            CHECK(crt::walk4_camera(e, eps));
            e[a] = sign * 24.f;
            CHECK(crt::walk4_camera(e, eps));
            e[a] = sign * std::nextafter(24.f, inf);
            CHECK(!crt::walk4_camera(e, eps));
            e[a] = sign * inf;
            CHECK(!crt::walk4_camera(e, eps));
            e[a] = nan;
            CHECK(!crt::walk4_camera(e, eps));
        }
    const float o[3] = {0.f, 0.f, 0.f};
    CHECK(crt::walk4_camera(o, 1.f) && !crt::walk4_camera(o, std::nextafter(1.f, inf)));  // range 2^20
    CHECK(crt::walk4_camera(o, std::ldexp(1.f, -41)) && !crt::walk4_camera(o, std::nextafter(std::ldexp(1.f, -41), 0.f)));
    CHECK(!crt::walk4_camera(o, nan) && !crt::walk4_camera(o, inf));
    return 0;
}
''')


def test_memory_a_call_can_do_without(tmp_path):
    """A refused optional buffer is no error, stays empty and takes nothing from what was reserved before it; it is
    there once memory is; growing frees before it allocates."""
    run_cpp(tmp_path, r'''
static size_t g_free = 0, g_live = 0;
struct Budget {
    static void* alloc(size_t n) {
        if (n > g_free) return nullptr;
        size_t* p = static_cast<size_t*>(std::malloc(sizeof(size_t)));
        *p = n;
        g_free -= n;
        ++g_live;
        return p;
    }
    static void free(void* p) { g_free += *static_cast<size_t*>(p); --g_live; std::free(p); }
};
using Buf = crt::GrowingBuffer<Budget>;
int main() {
    const size_t tree = Buf::wanted(1000), nodes = Buf::wanted(640);
    g_free = tree + nodes - 1;  // a build that just fits, without the optional nodes
    Buf a, b;
    CHECK(a.try_reserve(1000) && a.cap == tree);
    CHECK(!b.try_reserve(640) && b.p == nullptr && b.cap == 0 && g_live == 1);
    CHECK(a.p && a.try_reserve(1000) && g_live == 1);  // held, and not allocated again
    g_free += 1;
    CHECK(b.try_reserve(640) && b.p && g_free == 0);
    void* old = b.p;
    CHECK(b.try_reserve(b.cap) && b.p == old);
    a.release();
    CHECK(b.try_reserve(1000) && g_live == 1);  // out of what it and a gave back
    CHECK(!b.try_reserve(100000) && b.p == nullptr && g_live == 0 && g_free == tree + nodes);
    b.release();
    return 0;
}
''')


def test_rays_that_pay_for_the_compressed_nodes(tmp_path):
    run_cpp(tmp_path, r'''
using D = crt::Walk4Demand;
int main() {
    CHECK(crt::walk4_pays(D::closest(65536), 4194304) && !crt::walk4_pays(D::closest(65536), 4194305));
    CHECK(crt::walk4_pays(D::any(65536), 1048576) && !crt::walk4_pays(D::any(65536), 1048577));
    CHECK(crt::walk4_pays(D::pixels(262144), 1048576) && !crt::walk4_pays(D::pixels(262143), 1048576));
    CHECK(!crt::walk4_pays(3 * D::closest(65536), 16777216) && crt::walk4_pays(4 * D::closest(65536), 16777216));
    CHECK(crt::walk4_pays(D::closest(0xFFFFFFFFull), 0xFFFFFFFFu));  // no overflow at the largest calls
    return 0;
}
''')


def test_counting_up_to_the_largest_calls(tmp_path):
    """A persistent grid's tiles end for every 32-bit number of samples, and its ray counter never comes round."""
    run_cpp(tmp_path, r'''
int main() {
    CHECK(crt::tiles_of(0, 128) == 0 && crt::tiles_of(1, 128) == 1 && crt::tiles_of(128, 128) == 1 && crt::tiles_of(129, 128) == 2);
    for (uint32_t n : {0xFFFFFFFFu, 0xFFFFFF81u, 0xFFFFFF80u, 0xFFFFB400u, 0x80000001u}) {
        const uint32_t tiles = crt::tiles_of(n, 128);
        CHECK(128ull * tiles >= n && 128ull * (tiles - 1) < n);
        uint64_t steps = 0;
        uint32_t last = 0;
        for (uint32_t tile = 151; tile < tiles; tile += 152, ++steps) { CHECK(tile >= last); last = tile; }
        CHECK(steps == (tiles - 151 + 151) / 152);
    }
    CHECK(static_cast<uint64_t>(crt::kMostPoolItems) + 32ull * 152 * 64 < (1ull << 32));
    return 0;
}
''')
