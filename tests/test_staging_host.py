"""Staging ring: every launch reads the bytes that were staged for it, wherever the ring
wraps.  The header is compiled here with a fake device whose streams run as late, and
in as odd an order, as their events allow, so no GPU is needed; the library's context
uses the same code."""
import os
import shutil
import subprocess

import pytest

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(REPO, "hicma_parsec_b200", "csrc")

MAIN = r"""
#include <cstdio>
#include <cstdlib>
#include <deque>
#include <memory>
#include <random>
#include "staging.h"
using namespace tlr;

struct Ctx {
    Ring ring;
    int cur = 0;
    std::deque<std::function<bool()>> q[2];   // operations of two streams; false: its event is not there yet
    int wrong = 0;
    std::mt19937 rng;
    std::vector<char> h, d;
    explicit Ctx(size_t bytes, unsigned seed) : rng(seed), h(bytes), d(bytes) {
        ring.h = h.data(); ring.d = d.data(); ring.bytes = bytes;
    }
    bool step(int s) {
        if (q[s].empty() || !q[s].front()()) return false;
        q[s].pop_front();
        return true;
    }
    void some() { for (int n = rng() % 4; n > 0; --n) step(rng() & 1); }
    void drain(int s) { while (!q[s].empty()) if (!step(s)) { if (!step(1 - s)) abort(); } }
    int ring_upload(size_t off, size_t n) {
        q[cur].push_back([=] { std::memcpy(d.data() + off, h.data() + off, n); return true; });   // reads the host late
        some();
        return 0;
    }
    int ring_wait_current() { drain(cur); return 0; }
    int ring_wait_all() { drain(0); drain(1); return 0; }
    int kernel(std::vector<std::pair<const char *, std::vector<char>>> args) {
        q[cur].push_back([this, args] {
            for (auto &a : args) wrong += std::memcmp(a.first, a.second.data(), a.second.size()) != 0;
            return true;
        });
        some();
        return 0;
    }
    std::vector<char> array() {
        std::vector<char> v(1 + rng() % 700);
        for (char &x : v) x = (char)rng();
        return v;
    }
};

// a launch with one array, with two, or one on each stream between a fork and a join
static int launch(Ctx *c, int kind) {
    if (kind == 0) {
        const std::vector<char> a = c->array();
        const char *d = stage(c, a.data(), a.size());
        return d ? issue(c, [=] { return c->kernel({{d, a}}); }) : 1;
    }
    if (kind == 1) {
        const std::vector<char> a = c->array(), b = c->array();
        char *da, *db;
        if (!stage_both(c, a, b, &da, &db)) return 1;
        return issue(c, [=] { return c->kernel({{da, a}, {db, b}}); });
    }
    auto there = std::make_shared<std::vector<int>>(2, 0);   // the events: fork, join
    auto record = [=](int w) { c->q[c->cur].push_back([=] { (*there)[w] = 1; return true; }); return 0; };
    auto wait = [=](int w, int s) { c->q[s].push_back([=] { return (*there)[w] != 0; }); return 0; };
    if (issue(c, [=] { record(0); return wait(0, 1); })) return 1;
    for (int s : {0, 1}) {
        c->cur = s;
        const int rc = launch(c, c->rng() & 1);
        c->cur = 0;
        if (rc) return rc;
    }
    return issue(c, [=] { c->cur = 1; record(1); c->cur = 0; return wait(1, 0); });
}

int main(int argc, char **argv) {
    for (unsigned seed = 0; seed < 3000; ++seed) {
        Ctx c(2048 + 256 * (seed % 9), seed);
        for (int b = 0; b < 6; ++b) {
            if (c.rng() % 3 == 0) {
                for (int n = c.rng() % 5; n > 0; --n) if (launch(&c, c.rng() % 2)) return printf("refused\n"), 1;
                continue;
            }
            BatchOf<Ctx> batch(&c);
            for (int n = 1 + c.rng() % 14; n > 0; --n) if (launch(&c, c.rng() % 3)) return printf("refused\n"), 1;
            if (batch.flush()) return 1;
        }
        c.ring_wait_all();
        if (c.wrong) return printf("seed %u: %d launches read other bytes\n", seed, c.wrong), 1;
    }
    // two arrays of a launch without room made for both: refused at a wrap between them
    Ctx c(2048, 1);
    BatchOf<Ctx> batch(&c);
    char a[700] = {}, z[1100] = {};
    if (!stage(&c, a, sizeof a)) return 2;
    issue(&c, [] { return 0; });
    if (!stage(&c, a, sizeof a) || stage(&c, z, sizeof z)) return printf("a wrap before the launch was let through\n"), 1;
    return 0;
}
"""


def test_launches_read_what_was_staged_for_them(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    if not cxx:
        pytest.skip("no C++ compiler")
    (tmp_path / "main.cpp").write_text(MAIN)
    exe = str(tmp_path / "main")
    subprocess.run([cxx, "-std=c++17", "-O1", "-I", CSRC, str(tmp_path / "main.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout
