"""The copy threads of pageable transfers (host/hostcopy.cpp), compiled alone: every size arrives whole; no more
threads than OMP_NUM_THREADS; a process that cannot make threads, or is forked after the set-up's OpenMP loops
(one worker per device after a common set-up), still copies; and a child leaves a team of its parent alone.  Transfers at once have a team each; the threads end with the last
holder."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "rast-3dmhd_b200")

MAIN = r"""
#include <sys/resource.h>
#include <sys/wait.h>
#include <unistd.h>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <filesystem>
#include <iterator>
#include <memory>
#include <thread>
#include <vector>
#include "r3d_host.hpp"

static int threads() {
    return (int)std::distance(std::filesystem::directory_iterator("/proc/self/task"), {});
}
static std::vector<unsigned char> a(9u << 20), b(a.size());
static bool copies(r3db::CopyTeam& t) {
    for (size_t i = 0; i < a.size(); ++i) a[i] = (unsigned char)(i * 2654435761u >> 13);
    const size_t k = size_t(1) << 20;
    for (size_t n : {size_t(0), size_t(1), k - 1, k, k + 1, 3 * k + 7, size_t(8) << 20, a.size()}) {
        std::memset(b.data(), 0, b.size());
        t.copy(b.data(), a.data(), n);
        if (std::memcmp(a.data(), b.data(), n)) return false;
        for (size_t i = n; i < b.size(); ++i)
            if (b[i]) return false;
    }
    return true;
}
static int child(int (*f)(r3db::CopyTeam*), r3db::CopyTeam* t) {
    const pid_t p = fork();
    if (p == 0) {
        alarm(20);
        _exit(f(t));
    }
    int st = 0;
    waitpid(p, &st, 0);
    return WIFEXITED(st) ? WEXITSTATUS(st) : 100 + WTERMSIG(st);
}
int main(int, char** argv) {
    const int limit = std::atoi(argv[1]);
    std::vector<double> x(1 << 20);
#pragma omp parallel for
    for (long i = 0; i < (long)x.size(); ++i) x[i] = (double)i;  // the set-up's loops
    const int before = threads();
    auto* t = new r3db::CopyTeam;
    if (threads() - before > limit - 1) return 1;
    if (!copies(*t)) return 2;
    auto own = [](r3db::CopyTeam*) {
        r3db::CopyTeam c;
        return copies(c) ? 0 : 1;
    };
    auto parents = [](r3db::CopyTeam* p) {
        const bool ok = copies(*p);
        delete p;
        return ok ? 0 : 1;
    };
    auto poor = [](r3db::CopyTeam*) {  // no address space for a thread's stack
        std::FILE* f = std::fopen("/proc/self/statm", "r");
        long pages = 0;
        if (!f || std::fscanf(f, "%ld", &pages) != 1) return 3;
        std::fclose(f);
        rlimit r;
        getrlimit(RLIMIT_AS, &r);
        r.rlim_cur = (rlim_t)pages * sysconf(_SC_PAGESIZE) + (20u << 20);
        setrlimit(RLIMIT_AS, &r);
        std::unique_ptr<r3db::CopyTeam> c[8];
        for (auto& q : c) q.reset(new r3db::CopyTeam);  // 8 MB of stack each: most get none
        return copies(*c[7]) ? 0 : 1;
    };
    if (int rc = child(own, t)) return 10 + rc;
    if (int rc = child(parents, t)) return 30 + rc;
    if (int rc = child(poor, t)) return 50 + rc;
    delete t;

    const int alone = threads();
    auto pool = r3db::CopyTeams::get();
    if (pool != r3db::CopyTeams::get()) return 70;
    auto users = [](r3db::CopyTeam*) {  // transfers of two threads at once, then one after the other
        auto p = r3db::CopyTeams::get();
        std::vector<unsigned char> c(a.size()), d(a.size());
        auto run = [&](std::vector<unsigned char>& to) {
            for (int q = 0; q < 20; ++q) {
                r3db::CopyTeams::Use u(*p);
                u->wake();
                u->copy(to.data(), a.data() + q, a.size() - q);
                if (std::memcmp(to.data(), a.data() + q, a.size() - q)) to[0] = ~a[q], q = 20;
            }
            return 0;
        };
        std::thread other([&] { run(c); });
        run(d);
        other.join();
        return c[0] == a[19] && d[0] == a[19] ? 0 : 1;
    };
    if (int rc = users(nullptr)) return 70 + rc;
    if (threads() - alone > 2 * (limit - 1)) return 73;
    if (int rc = child(users, nullptr)) return 80 + rc;  // the parent's teams are none of the child's
    pool.reset();
    return threads() == alone ? 0 : 90;
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("hostcopy")
    (d / "main.cpp").write_text(MAIN)
    subprocess.run(["g++", "-O2", "-std=c++17", "-fopenmp", "-I", os.path.join(PKG, "host"), "-I",
                    os.path.join(ROOT, "include"), str(d / "main.cpp"), os.path.join(PKG, "host", "hostcopy.cpp"),
                    "-o", str(d / "run"), "-pthread"], check=True)
    return str(d / "run")


@pytest.mark.parametrize("limit", [1, 2, 8])
def test_copy_team(program, limit):
    env = dict(os.environ, OMP_NUM_THREADS=str(limit))
    r = subprocess.run([program, str(limit)], env=env, timeout=120)
    assert r.returncode == 0
