"""Memory of the wide core SVD for every width: each part lies inside the shared
memory or scratch that is reserved for it and beside the parts alive with it.  The
header with the arithmetic is compiled here, so no GPU is needed; the kernel and its
launcher use the same functions."""
import os
import shutil
import subprocess

import pytest

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(REPO, "hicma_parsec_b200", "csrc")

MAIN = r"""
#include <cstdio>
#include <vector>
#include "core_layout.h"
using namespace tlr;
struct Part { const char *name; size_t at, n; };   // doubles
static int check(int K, int cs, const char *what, size_t limit, const std::vector<Part> &v) {
    for (size_t i = 0; i < v.size(); ++i) {
        if (v[i].at + v[i].n > limit) {
            printf("K %d, %d CTAs: %s: %s ends at %zu of %zu\n", K, cs, what, v[i].name, v[i].at + v[i].n, limit);
            return 1;
        }
        for (size_t j = 0; j < i; ++j)
            if (v[i].at < v[j].at + v[j].n && v[j].at < v[i].at + v[i].n) {
                printf("K %d, %d CTAs: %s: %s over %s\n", K, cs, what, v[i].name, v[j].name);
                return 1;
            }
    }
    return 0;
}
// a task of K columns in a launch whose widest has kmax, laid out as `place` says
static int task(int K, int cs, int place, size_t bytes, size_t limit) {
    const bool hv = place & W_HV_SHARED, t = place & W_T_SHARED;
    const size_t k = (size_t)K, ncl = (size_t)wide_ncl(K, cs), sm = bytes / 8, work = wide_work_doubles(K, limit);
    std::vector<Part> qr_sm, qr_work, sort_sm, sort_work;
    qr_work = {{"X", 0, k * k}, {"sigma", wide_layout(K, cs, 0, place).sig, k}, {"flags", wide_layout(K, cs, 0, place).flags, 64}};
    sort_work = {{"X", 0, k * (k + WP)}, qr_work[1], qr_work[2]};
    const size_t csr = (size_t)(cs < K ? cs : K);
    for (size_t r = 0; r < csr; ++r) {
        const WideLayout w = wide_layout(K, cs, (int)r, place);
        if (!hv) qr_work.push_back({"hv", w.hv, k});
        if (!t) {
            qr_work.push_back({"T", w.T, ncl * k});
            sort_work.push_back({"sorted values", w.sort, k + (k + 1) / 2});
        }
    }
    const WideLayout w = wide_layout(K, cs, cs - 1, place);
    qr_sm = {{"sigl", w.sigl, ncl}};
    if (hv) qr_sm.push_back({"hv", w.hv, k});
    if (t) qr_sm.push_back({"T", w.T, ncl * k}), sort_sm = {{"sorted values", w.sort, k + (k + 1) / 2}};
    return check(K, cs, "QR", sm, qr_sm) | check(K, cs, "QR scratch", work, qr_work) | check(K, cs, "sort", sm, sort_sm) |
           check(K, cs, "sort scratch", work, sort_work) |
           check(K, cs, "Jacobi", sm, {{"G", 0, WP * WLD}, {"J", WP * WLD, WP * WLD}, {"partials", 2 * WP * WLD, W_NW * W_TILES * 64}});
}
int main() {
    int bad = 0, seen = 0;
    for (size_t limit : {W_SMEM_MAX, (size_t)100000, (size_t)0})
        for (int kmax = 65; kmax <= 40000 && !bad; kmax += kmax < 9000 ? 1 : 37)
            for (int cs : {4, 8, 16}) {
                if (cs != wide_cluster(kmax) && !(cs == 8 && wide_cluster(kmax) == 16)) continue;   // 16 falls back to 8
                const int place = wide_place(kmax, cs, limit);
                const size_t bytes = wide_smem(kmax, cs, place);
                seen |= 1 << place;
                if (bytes > W_SMEM_MAX) { printf("K %d: %zu bytes\n", kmax, bytes); return 1; }
                // the narrowest, a middle and the widest core that this launch can hold
                const int lo = kmax <= W_EDGE1 ? 65 : kmax <= W_EDGE2 ? W_EDGE1 + 1 : W_EDGE2 + 1;
                for (int K : {lo, (lo + kmax) / 2, kmax}) bad |= task(K, cs, place, bytes, limit);
            }
    if (seen != ((1 << 0) | (1 << W_HV_SHARED) | (1 << (W_HV_SHARED | W_T_SHARED)))) { printf("places %x\n", seen); return 1; }
    return bad;
}
"""


def test_every_width_stays_inside_its_memory(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    if not cxx:
        pytest.skip("no C++ compiler")
    (tmp_path / "main.cpp").write_text(MAIN)
    exe = str(tmp_path / "main")
    subprocess.run([cxx, "-std=c++17", "-O1", "-I", CSRC, str(tmp_path / "main.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout
