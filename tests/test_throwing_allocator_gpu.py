"""A null-space allocator that throws: the exception leaves the C entry point,
and the thread's page-locked words are back in its hands."""
import os
import subprocess

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include <cstdio>
#include <cstdint>
#include <cstring>
#include <stdexcept>
#include <vector>
#include <unistd.h>
#include "mela.h"
static long rss_kb() {
    long a = 0, b = 0;
    FILE *f = fopen("/proc/self/statm", "r");
    if (!f || fscanf(f, "%ld %ld", &a, &b) != 2) return -1;
    fclose(f);
    return b * (sysconf(_SC_PAGESIZE) / 1024);
}
static uint8_t *thrower(void *, int64_t, int64_t) { throw std::runtime_error("no room"); }
static uint8_t *keeper(void *ctx, int64_t r, int64_t c) {
    auto *v = (std::vector<uint8_t> *)ctx;
    v->assign((size_t)(r * c), 7);
    return v->data();
}
int main() {
    const int m = 40, n = 90;
    std::vector<uint8_t> a(m * n), z;
    for (int i = 0; i < m * n; ++i) a[i] = (uint8_t)((i * 2654435761u >> 13) & 1);
    mela_host_matrix M{MELA_KIND_LOGICAL, 0, m, n, a.data()};
    int64_t f = 0;
    int caught = 0;
    auto one = [&] {
        try {
            mela_null_gf2(&M, thrower, nullptr, &f);
        } catch (const std::runtime_error &) {
            ++caught;
        }
    };
    for (int i = 0; i < 5; ++i) one();
    const long before = rss_kb();
    for (int i = 0; i < 60; ++i) one();
    const long grown = rss_kb() - before;
    if (mela_null_gf2(&M, keeper, &z, &f) != MELA_OK) return 2;
    for (int i = 0; i < m; ++i)
        for (int64_t c = 0; c < f; ++c) {
            int s = 0;
            for (int j = 0; j < n; ++j) s ^= a[i + j * m] & z[j + c * n];
            if (s) return 3;
        }
    printf("caught %d grown %ld KB nullity %lld\n", caught, grown, (long long)f);
    return caught == 65 && grown < 6000 && f >= n - m ? 0 : 4;
}
"""


def test_allocator_that_throws(cuda, tmp_path):
    src, exe = tmp_path / "thrower.cpp", tmp_path / "thrower"
    src.write_text(PROGRAM)
    pkg = os.path.join(ROOT, "mex_linear_algebra_b200")
    subprocess.run(["g++", "-std=c++17", "-I" + os.path.join(ROOT, "include"), str(src), "-o", str(exe),
                    os.path.join(pkg, "libmela_b200.so"), "-Wl,-rpath," + pkg], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
