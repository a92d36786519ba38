"""The threads of the spin transfers (espins_gb300/csrc/esp_copy.h), through a
small program compiled with g++: every value is converted once whatever the
number of users and threads, the threads are started beside the users and kept
between them, given back when idle, and a forked child neither has nor waits
for them."""
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "espins_gb300", "csrc")

PROGRAM = r'''
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <dirent.h>
#include <sys/wait.h>
#include "esp_copy.h"
using namespace esp;
static int tasks()
{
    int n = 0;
    DIR *d = opendir("/proc/self/task");
    while (dirent *e = readdir(d)) n += e->d_name[0] != '.';
    closedir(d);
    return n;
}
static void nap(int ms) { std::this_thread::sleep_for(std::chrono::milliseconds(ms)); }
// a transfer to the ring and one back, drained chunk by chunk as the spins are
static bool transfer(CopyPool *pool, long long total, unsigned seed)
{
    std::vector<double> in(total), out(total, -1.0);
    std::vector<float> want(total);
    for (long long i = 0; i < total; ++i) {
        seed = seed * 1664525u + 1013904223u;
        in[i] = (double)(int)seed * 1.2345678901234567e-3;
        want[i] = (float)in[i];
    }
    const long long chunk = 4 * kCopyPiece;
    const int ring = 3;
    const long long n = (total + chunk - 1) / chunk;
    std::vector<float> r(ring * chunk), got(total);
    {
        CopyJob job(true, in.data(), r.data(), total, chunk, ring);
        job.open(ring);
        CopyTeam team(pool, job);
        for (long long c = 0; c < n; ++c) {
            job.finish(c);
            std::memcpy(&got[c * chunk], &r[c % ring * chunk], sizeof(float) * std::min(chunk, total - c * chunk));
            job.open(c + ring + 1);
        }
    }
    if (std::memcmp(got.data(), want.data(), sizeof(float) * total)) return false;
    {
        CopyJob job(false, out.data(), r.data(), total, chunk, ring);
        CopyTeam team(pool, job);
        for (long long c = 0; c < n; ++c) {
            if (c >= ring) job.finish(c - ring);
            std::memcpy(&r[c % ring * chunk], &want[c * chunk], sizeof(float) * std::min(chunk, total - c * chunk));
            job.open(c + 1);
        }
        for (long long c = std::max(0LL, n - ring); c < n; ++c) job.finish(c);
    }
    for (long long i = 0; i < total; ++i)
        if (out[i] != (double)want[i]) return false;
    return true;
}
#define CHECK(c) do { if (!(c)) { std::printf("line %d: %s\n", __LINE__, #c); return 1; } } while (0)
int main(int argc, char **argv)
{
    const std::string_view what = argv[1];
    const int most = (int)std::min(15u, std::max(1u, std::thread::hardware_concurrency()) - 1);
    if (what == "convert") {
        CopyPool pool;
        for (long long total : {1LL, 16384LL, 65536LL, 65537LL, 300001LL, 2000003LL})
            for (int k = 0; k < 3; ++k) CHECK(transfer(&pool, total, 7 * k + (unsigned)total));
        CHECK(transfer(nullptr, 300001, 5));
        std::atomic<int> bad{0};
        std::vector<std::thread> users;
        for (int u = 0; u < 6; ++u)
            users.emplace_back([&, u] {
                for (int k = 0; k < 20; ++k)
                    if (!transfer(&pool, 100000 + 50000 * u + k, u + 10 * k)) ++bad;
            });
        for (std::thread &t : users) t.join();
        CHECK(bad == 0);
    } else if (what == "kept") {
        const int t0 = tasks();
        CopyPool *pool = CopyPool::get();
        pool->reserve(1000);
        CHECK(tasks() == t0);                     // too small for a helper
        pool->reserve(10 << 20);
        for (int k = 0; k < 200 && tasks() < t0 + most; ++k) nap(5);
        CHECK(tasks() == t0 + most);
        CHECK(transfer(pool, 2000003, 3) && CopyPool::get() == pool);
        CHECK(tasks() == t0 + most);
    } else if (what == "idle") {
        const int t0 = tasks();
        CopyPool pool(std::chrono::milliseconds(30));
        for (int round = 0; round < 3; ++round) {
            pool.reserve(10 << 20);
            CHECK(transfer(&pool, 2000003, round));
            for (int k = 0; k < 400 && tasks() > t0; ++k) nap(5);
            CHECK(tasks() == t0);                 // given back
        }
        pool.reserve(10 << 20);                   // destroyed while they start
    } else if (what == "fork") {
        CopyPool *pool = CopyPool::get();
        pool->reserve(10 << 20);
        for (int k = 0; k < 200 && tasks() < 1 + most; ++k) nap(5);
        const pid_t child = fork();
        if (!child) {
            if (!transfer(pool, 300001, 1)) std::_Exit(2);
            std::exit(0);                         // with its exit handlers
        }
        int status = -1;
        for (int k = 0; k < 1000; ++k) {
            if (waitpid(child, &status, WNOHANG) == child) break;
            status = -1;
            nap(10);
        }
        if (status == -1) kill(child, 9);
        CHECK(status == 0);
        CHECK(transfer(pool, 2000003, 9));
    }
    return 0;
}
'''


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("copy")
    src, exe = d / "copy.cpp", d / "copy"
    src.write_text("#include <string_view>\n#include <signal.h>\n" + PROGRAM)
    subprocess.run(["g++", "-O1", "-g", "-std=c++17", "-pthread", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    return str(exe)


@pytest.mark.parametrize("what", ["convert", "kept", "idle", "fork"])
def test_copy_pool(program, what):
    r = subprocess.run([program, what], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
