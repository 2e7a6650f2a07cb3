"""Device memory kept for the next descriptors: what is handed out never overlaps what
is in use, what is kept is bounded, and it all goes back on a failed allocation and
with the last context.  The header is compiled here on a fake allocator, so no GPU is
needed; the library uses it on cudaMalloc."""
import os
import shutil
import subprocess

import pytest

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(REPO, "hicma_parsec_b200", "csrc")

MAIN = r"""
#include <atomic>
#include <cstdio>
#include <random>
#include <thread>
#include <vector>
#include "regions.h"
using namespace tlr;

static const size_t MB = 1 << 20, DEVICE = 4096 * MB;
struct Fake {
    static std::mutex mu;
    static std::map<char *, size_t> live;      // addresses only, nothing is touched
    static size_t used;
    static long allocs;
    static char *next;
    static int alloc(void **p, size_t n) {
        std::lock_guard<std::mutex> lk(mu);
        if (used + n > DEVICE) return 2;
        ++allocs;
        used += n;
        *p = next;
        next += n;
        live[(char *)*p] = n;
        return 0;
    }
    static bool is_oom(int e) { return e == 2; }
    static void release(void *p) {
        std::lock_guard<std::mutex> lk(mu);
        auto f = live.find((char *)p);
        if (f == live.end()) { printf("released twice\n"); std::_Exit(1); }
        used -= f->second;
        live.erase(f);
    }
};
std::mutex Fake::mu;
std::map<char *, size_t> Fake::live;
size_t Fake::used = 0;
long Fake::allocs = 0;
char *Fake::next = (char *)0x100000000;

#define REQUIRE(x) do { if (!(x)) { printf("line %d: %s\n", __LINE__, #x); std::_Exit(1); } } while (0)

int main() {
    Regions<Fake> r;
    const size_t limit = 1024 * MB;
    r.enter(limit);
    void *a, *b, *c;
    // the same size again, and one that is a little smaller: no new allocation
    REQUIRE(!r.take(&a, 100 * MB) && !r.take(&b, 3));
    const long n0 = Fake::allocs;
    r.give(a, true);
    REQUIRE(r.held() == 100 * MB);
    REQUIRE(!r.take(&c, 85 * MB) && c == a && Fake::allocs == n0 && r.held() == 0);
    // much smaller or larger ones are not served by it
    r.give(c, true);
    REQUIRE(!r.take(&c, 40 * MB) && c != a && !r.take(&a, 101 * MB) && Fake::allocs == n0 + 2);
    r.give(a, true), r.give(c, true);
    // after an error of the device a region is not kept
    size_t h = r.held();
    REQUIRE(!r.take(&a, 300 * MB));
    r.give(a, false);
    REQUIRE(r.held() == h);
    // bounded, the oldest first; one above the bound is not kept
    std::vector<void *> v(10);
    for (auto &p : v) REQUIRE(!r.take(&p, 200 * MB));
    for (auto &p : v) { r.give(p, true); REQUIRE(r.held() <= limit); }
    REQUIRE(r.held() == limit - 24 * MB);
    for (int q = 9; q >= 5; --q) REQUIRE(!r.take(&a, 200 * MB) && (a == v[5] || a == v[6] || a == v[7] || a == v[8] || a == v[9]));
    r.trim();
    for (int q = 5; q < 10; ++q) r.give(v[q], true);
    REQUIRE(!r.take(&a, 2000 * MB));
    h = r.held();
    r.give(a, true);
    REQUIRE(r.held() == h);
    // a failing allocation gets what is kept
    REQUIRE(r.held() == 1000 * MB && !r.take(&a, 3500 * MB) && r.held() == 0);
    REQUIRE(r.take(&c, 1000 * MB) == 2 && c == nullptr);
    r.give(a, true);
    // many small regions
    std::vector<void *> s(1000);
    for (auto &p : s) REQUIRE(!r.take(&p, 100));
    for (auto &p : s) r.give(p, true);
    REQUIRE(Fake::live.size() <= 256 + 1);      // and b
    // a second context: the last one to leave gives it back
    r.enter(limit);
    r.leave();
    REQUIRE(r.held() > 0);
    // threads: regions in use at the same time never overlap
    std::mutex mu;
    std::map<char *, size_t> busy;
    std::atomic<int> bad{0};
    auto work = [&](int seed) {
        std::mt19937 g(seed);
        for (int q = 0; q < 20000; ++q) {
            const size_t n = 1 + g() % (60 * MB);
            void *p;
            if (r.take(&p, n)) continue;
            {
                std::lock_guard<std::mutex> lk(mu);
                auto it = busy.lower_bound((char *)p);
                if (it != busy.end() && it->first < (char *)p + n) ++bad;
                if (it != busy.begin()) { --it; if (it->first + it->second > (char *)p) ++bad; }
                busy[(char *)p] = n;
            }
            std::this_thread::yield();
            {
                std::lock_guard<std::mutex> lk(mu);
                busy.erase((char *)p);
            }
            r.give(p, g() % 50 != 0);
        }
    };
    std::vector<std::thread> t;
    for (int q = 0; q < 4; ++q) t.emplace_back(work, q);
    for (auto &x : t) x.join();
    REQUIRE(bad == 0);
    r.give(b, true);
    r.leave();
    REQUIRE(r.held() == 0 && Fake::used == 0 && Fake::live.empty());
    return 0;
}
"""


def test_regions_are_bounded_and_never_shared(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    if not cxx:
        pytest.skip("no C++ compiler")
    (tmp_path / "main.cpp").write_text(MAIN)
    exe = str(tmp_path / "main")
    subprocess.run([cxx, "-std=c++17", "-O1", "-pthread", "-I", CSRC, str(tmp_path / "main.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout
