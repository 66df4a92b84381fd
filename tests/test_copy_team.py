"""The threads of large host copies (abt_b200/csrc/copy_team.h), without a GPU: every byte arrives,
whatever the size, from several teams at once; no more threads than the processors the caller is
bound to, OpenMP's limit and an enclosing parallel region allow; and none for a while when one
of them held a copy up (rests of 256, 512, ... copies: at most four such copies in 2,000)."""
import os
import subprocess

import pytest

from tests.conftest import ROOT

SOURCE = r"""
#include <dirent.h>
#include <stdio.h>
#include <stdlib.h>
#include <time.h>
#include "copy_team.h"
#include <atomic>
#include <thread>
#include <vector>
using pbt::CopyTeam;
static int tasks() {
    int n = 0;
    DIR *d = opendir("/proc/self/task");
    while (readdir(d)) n++;
    closedir(d);
    return n - 2;
}
static bool copies(unsigned seed) {
    CopyTeam p;
    bool ok = true;
    const size_t most = 5u << 20;
    std::vector<char> a(most), b(most);
    for (size_t i = 0; i < most; i++) a[i] = (char)(i * 2654435761u >> 13) + (char)seed;
    const size_t K = CopyTeam::kPiece;
    const size_t sizes[] = {0, 1, K - 1, K, K + 1, 7 * K, 8 * K, 8 * K + 1, 512u << 10, most};
    for (int rep = 0; rep < 200; rep++) {
        p.begin();
        for (int chunk = 0; chunk < 4; chunk++) {
            const size_t n = sizes[(rep + 3 * chunk + seed) % 10], o = (rep * 131 + chunk) % 64;
            const size_t m = n > most - 64 ? most - 64 : n;
            std::fill(b.begin(), b.end(), 0);
            p.run(b.data() + o, a.data() + o, m);
            ok = ok && !memcmp(b.data() + o, a.data() + o, m) && (o + m >= most || b[o + m] == 0) && (!o || !b[o - 1]);
        }
        p.end();
    }
    return ok;
}
static std::thread::id owner;
static std::atomic<bool> held;
static void slow(char *d, const char *s, size_t n) {
    memcpy(d, s, n);
    if (std::this_thread::get_id() == owner) return;
    held = true;
    struct timespec w = {0, 6000000};
    nanosleep(&w, nullptr);
}
int main() {
    printf("allowed %d\n", CopyTeam::allowed());
    const int before = tasks();
    {
        CopyTeam p;
        std::vector<char> a(1 << 20), b(1 << 20);
        p.begin();
        p.run(b.data(), a.data(), a.size());
        p.end();
        printf("started %d\n", tasks() - before);
    }
    int inside = -1;
#pragma omp parallel num_threads(2)
#pragma omp master
    inside = omp_get_num_threads() > 1 ? CopyTeam::allowed() : 1;
    printf("inside %d\n", inside);
    {
        // threads that lose their core within a piece (here: sleep in it)
        CopyTeam p(slow);
        std::vector<char> a(1 << 20, 7), b(1 << 20);
        owner = std::this_thread::get_id();
        int with = 0;
        bool same = true;
        for (int c = 0; c < 2000; c++) {
            held = false;
            std::fill(b.begin(), b.end(), 0);
            p.begin();
            for (int k = 0; k < 2; k++) p.run(b.data() + k * (512 << 10), a.data() + k * (512 << 10), 512 << 10);
            p.end();
            same = same && a == b;
            with += held;
        }
        printf("held %d\nsame %d\n", with <= 4, same);
    }
    bool ok[4];
    std::vector<std::thread> t;
    for (int k = 0; k < 4; k++) t.emplace_back([&ok, k] { ok[k] = copies(k); });
    for (auto &x : t) x.join();
    printf("ok %d\n", ok[0] && ok[1] && ok[2] && ok[3]);
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("copy_team")
    (d / "t.cpp").write_text(SOURCE)
    subprocess.run(["g++", "-O2", "-std=c++17", "-fopenmp", "-pthread", "-I" + os.path.join(ROOT, "abt_b200", "csrc"),
                    str(d / "t.cpp"), "-o", str(d / "t")], check=True, capture_output=True)
    return str(d / "t")


@pytest.mark.parametrize("omp", [None, 1, 3])
@pytest.mark.parametrize("bound", [False, True])
def test_team(program, omp, bound):
    cpus = sorted(os.sched_getaffinity(0))
    env = {k: v for k, v in os.environ.items() if not k.startswith("OMP_")}
    if omp:
        env["OMP_NUM_THREADS"] = str(omp)
    r = subprocess.run([program], env=env, capture_output=True, text=True, timeout=300, check=True,
                       preexec_fn=(lambda: os.sched_setaffinity(0, cpus[:1])) if bound else None)
    got = dict(line.split() for line in r.stdout.splitlines())
    want = min(1 if bound else len(cpus), omp or len(cpus), 8)
    assert got == {"allowed": str(want), "inside": "1", "started": str(want - 1), "ok": "1", "held": "1", "same": "1"}
