"""The host BVH build keeps to the threads it is given - one limit for every build of the process - and its tree
does not depend on them.  A small program is linked to the builder; it counts the threads that are alive at once."""
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "cortexraytracercuda_b200" / "csrc"

MAIN = r"""
#include <dlfcn.h>
#include <pthread.h>
#include <atomic>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <thread>
#include "bvh_build.h"
static std::atomic<int> live{0}, most{0};
struct Arg { void* (*f)(void*); void* a; };
static void* run(void* p) {
    Arg g = *(Arg*)p;
    delete (Arg*)p;
    int n = ++live, m = most;
    while (n > m && !most.compare_exchange_weak(m, n)) {}
    void* r = g.f(g.a);
    --live;
    return r;
}
extern "C" int pthread_create(pthread_t* t, const pthread_attr_t* at, void* (*f)(void*), void* a) {
    static auto real = (int (*)(pthread_t*, const pthread_attr_t*, void* (*)(void*), void*))dlsym(RTLD_NEXT, "pthread_create");
    return real(t, at, run, new Arg{f, a});
}
static rtc::BvhInput boxes(size_t n) {
    rtc::BvhInput in;
    in.boxes.resize(n);
    srand(7);
    for (size_t i = 0; i < n; ++i) {
        const double u = rand() / (double)RAND_MAX * 6.283, z = rand() / (double)RAND_MAX * 2 - 1, r = sqrt(1 - z * z);
        const float c[3] = {(float)(r * cos(u)), (float)z, (float)(r * sin(u))};
        for (int k = 0; k < 3; ++k) { in.boxes[i].lo[k] = c[k] - 0.01f; in.boxes[i].hi[k] = c[k] + 0.01f; }
    }
    return in;
}
static rtc::BvhOutput tree(const rtc::BvhInput& in, int threads) {
    rtc::BvhOutput o;
    const char* err = nullptr;
    if (!rtc::build_bvh(in, 4, threads, o, &err)) exit(2);
    return o;
}
static bool same(const rtc::BvhOutput& a, const rtc::BvhOutput& b) {
    return a.nodes.size() == b.nodes.size() && !memcmp(a.nodes.data(), b.nodes.data(), a.nodes.size() * 4) &&
           a.order == b.order && a.nodes8.size() == b.nodes8.size() &&
           !memcmp(a.nodes8.data(), b.nodes8.data(), a.nodes8.size() * sizeof(a.nodes8[0])) && a.items8 == b.items8;
}
int main() {
    const rtc::BvhInput in = boxes(150000);
    const rtc::BvhOutput one = tree(in, 1);
    printf("1 %d\n", most.load());
    bool ok = true;
    for (int threads : {2, 3, 8, 0}) {
        most = 0;
        ok = same(tree(in, threads), one) && ok;
        printf("%d %d\n", threads ? threads : 4 * (int)std::thread::hardware_concurrency(), most.load());
    }
    most = 0;   // four builds at once, on four threads of their own
    std::thread t[4];
    bool oks[4];
    for (int k = 0; k < 4; ++k) t[k] = std::thread([&, k] { oks[k] = same(tree(in, 3), one); });
    for (int k = 0; k < 4; ++k) { t[k].join(); ok = ok && oks[k]; }
    printf("%d %d\n", 3 + 4, most.load());
    return ok ? 0 : 1;
}
"""


def test_threads_are_bounded_and_trees_equal(tmp_path):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("no g++")
    from cortexraytracercuda_b200.build import CXX_FLAGS
    (tmp_path / "main.cpp").write_text(MAIN)
    exe = tmp_path / "threads"
    subprocess.run([gxx, *CXX_FLAGS, "-w", str(tmp_path / "main.cpp"), str(CSRC / "bvh_build.cpp"), "-o", str(exe), "-lpthread",
                    "-ldl"], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr   # the same tree for every number of threads
    for line in r.stdout.splitlines():
        allowed, most = map(int, line.split())
        assert most <= allowed - 1, r.stdout        # threads beside the caller's
