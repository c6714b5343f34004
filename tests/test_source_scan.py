"""qp3d::scan_source_volumes, the scan of one load's or one batch's source
volumes: the lists are those of sequential scans, for volumes of several slabs,
of one, of one plane and without a sample; and one large volume is shared by the
host threads however many volumes the call has (counted by the threads that
the process had at the most)."""
import os
import subprocess

import pytest

import qp3d

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SRC = r'''
#include <atomic>
#include <chrono>
#include <cstdio>
#include <cstring>
#include <thread>
#include <vector>
#include "qp3d_internal.h"
using namespace qp3d;
struct Vol { int nx, ny, nz; std::vector<float> v; std::vector<SrcEntry> got; };
static int threads()
{
    FILE *f = fopen("/proc/self/status", "r");
    char line[256];
    int n = 0;
    while (fgets(line, sizeof(line), f)) if (sscanf(line, "Threads: %d", &n) == 1) break;
    fclose(f);
    return n;
}
int main()
{
    const int shape[][3] = {{320, 250, 240}, {37, 29, 53}, {2200, 2101, 1}, {16, 16, 16}};
    std::vector<Vol> vols;
    unsigned s = 12345u;
    for (auto &d : shape) {
        Vol v{d[0], d[1], d[2], std::vector<float>((size_t)d[0] * d[1] * d[2], 0.0f), {}};
        if (d[0] != 16)
            for (float &f : v.v) {
                s = s * 1664525u + 1013904223u;
                if ((s >> 20) < 3) f = (float)(s & 0xffff) - 30000.0f;
            }
        vols.push_back(std::move(v));
    }
    std::vector<SourceVolume> in;
    for (Vol &v : vols) in.push_back({v.v.data(), v.nx, v.ny, v.nz, &v.got});
    scan_source_volumes(in);
    for (Vol &v : vols) {
        size_t k = 0;
        for (int z = 0; z < v.nz; ++z)
            for (int x = 0; x < v.nx; ++x)
                for (int y = 0; y < v.ny; ++y) {
                    const float f = v.v[((size_t)z * v.nx + x) * v.ny + y];
                    if (f == 0.0f) continue;
                    if (k >= v.got.size() || v.got[k].x != x || v.got[k].y != y ||
                        v.got[k].z != z || v.got[k].v != f) return 1;
                    ++k;
                }
        if (k != v.got.size()) return 2;
    }
    // threads of a scan of one large volume beside a small one
    std::atomic<bool> done{false};
    std::atomic<int> most{0};
    const int before = threads();
    std::thread watch([&] {
        while (!done) { const int n = threads(); if (n > most) most = n; }
    });
    for (int r = 0; r < 20; ++r) scan_source_volumes({in[0], in[3]});
    done = true;
    watch.join();
    printf("%d %u\n", most - before - 1, std::thread::hardware_concurrency());
    return 0;
}
'''


def test_lists_and_threads(tmp_path):
    src = tmp_path / "scan.cpp"
    src.write_text(SRC)
    lib, exe = os.path.dirname(qp3d.LIB_PATH), str(tmp_path / "scan")
    r = subprocess.run(["g++", "-std=c++17", "-O2", "-I",
                        os.path.join(ROOT, "gpu-c_3dqmodeling_gb300", "csrc"), "-I",
                        os.path.join(ROOT, "include"), "-I", "/usr/local/cuda/include", str(src),
                        "-o", exe, "-L" + lib, "-lqp3d", "-lpthread", "-Wl,-rpath," + lib],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    out = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, (out.returncode, out.stdout)
    extra, hw = (int(t) for t in out.stdout.split())
    # five slabs, so up to four more threads; one thread a volume would start one
    assert extra >= min(2, hw - 1)
