"""The simulation's transforms on the CPU: csrc/simfft.cuh compiled with g++
against stand-ins for CUDA's names, the threads of a block run one after
another from barrier to barrier.  Every access to shared memory is checked: no
entry may be written by one thread and touched by another between two
barriers, none may lie outside the array.  The results are compared with the
transform's sum in 64 bits.

Tolerance: a stage rounds a value a few times (a direct sum of p terms p / 2
times, errors adding like a random walk): u = 6e-8 times 12 stages times
sqrt(113 / 2) is 5e-6 relative to the largest value's scale."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "waveforminversionust_b200", "csrc")

# what simfft.cuh takes from CUDA and from the file it includes
SHIM = r"""
#pragma once
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <ucontext.h>
#include <vector>
#define __device__
#define __host__
#define __forceinline__ inline
#define __noinline__
#define __constant__
#define __shared__
#define __align__(n)
struct Index { int x; };
inline Index threadIdx{0}, blockDim{0};
struct float2;
void note(const float2 *at, bool write);
struct float2 {
    float x, y;
    float2() : x(0), y(0) {}
    constexpr float2(float a, float b) : x(a), y(b) {}
    float2(const float2 &o) : x(o.x), y(o.y) { note(&o, false); }
    float2 &operator=(const float2 &o) {
        note(&o, false);
        note(this, true);
        x = o.x;
        y = o.y;
        return *this;
    }
};
inline float2 make_float2(float x, float y) { return float2(x, y); }
using std::max;
using std::min;
void __syncthreads();
namespace wust {
inline float2 cmul(float2 a, float2 b) { return float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x); }
}
"""

MAIN = r"""
#include "simfft.cuh"
using namespace wust;
constexpr int kRoom = 40000;
namespace wust { namespace sim { float2 fft_sm[kRoom]; } }
struct Cell { int wrote = -1, writer = -1, read = -1, reader = -1; };
static Cell cells[kRoom];
static int phase = 0, room = 0, races = 0, outside = 0;
void note(const float2 *at, bool write) {
    const long i = at - sim::fft_sm;
    if (at < sim::fft_sm || at >= sim::fft_sm + kRoom) return;          // registers
    if (i >= room) { ++outside; return; }
    Cell &c = cells[i];
    const int t = threadIdx.x;
    const bool written = c.wrote == phase && c.writer != t, read = c.read == phase && c.reader != t;
    if (written || (write && read)) ++races;
    if (write) { c.wrote = phase; c.writer = t; }
    else { c.reader = c.read == phase && c.reader != t ? -2 : t; c.read = phase; }
}
// the threads of a block as fibers, each run to its next barrier in turn
static ucontext_t scheduler;
static std::vector<ucontext_t> fibers;
static std::vector<char> finished;
static void (*body)();
void __syncthreads() { swapcontext(&fibers[threadIdx.x], &scheduler); }
static void run_one() {
    body();
    finished[threadIdx.x] = 1;
    swapcontext(&fibers[threadIdx.x], &scheduler);
}
static void run_block(int threads, void (*f)()) {
    static std::vector<std::vector<char>> stacks;
    while ((int)stacks.size() < threads) stacks.emplace_back(1 << 16);
    body = f;
    blockDim.x = threads;
    fibers.assign(threads, ucontext_t());
    finished.assign(threads, 0);
    for (int t = 0; t < threads; ++t) {
        getcontext(&fibers[t]);
        fibers[t].uc_stack.ss_sp = stacks[t].data();
        fibers[t].uc_stack.ss_size = stacks[t].size();
        fibers[t].uc_link = &scheduler;
        makecontext(&fibers[t], run_one, 0);
    }
    for (int done = 0; done < threads; ++phase) {
        for (int t = 0; t < threads; ++t) {
            if (finished[t]) continue;
            threadIdx.x = t;
            swapcontext(&scheduler, &fibers[t]);
            done += finished[t];
        }
        if (done && done < threads) { std::puts("threads part at a barrier"); std::exit(2); }
    }
    threadIdx.x = 0;
}
static int kind, n, lines, z0, plane;
static bool in_time;
template <class Lines> static void both(const Lines &l) {
    if (in_time) sim::fft_lines<true>(z0, l, 0, 0);
    else sim::fft_lines<false>(z0, l, 0, 0);
}
static sim::GridLines grid() { return kind ? sim::GridLines{lines, n | 1, 1, 1.f / lines} : sim::GridLines{lines, 1, lines, 1.f / lines}; }
static void transform() {
    if (kind == 2) both(sim::TileLines<2>{lines >> 2, plane});
    else if (kind == 3) both(sim::TileLines<3>{lines >> 3, plane});
    else both(grid());
}
static int place(int l, int e) {
    if (kind == 2) { const sim::TileLines<2> t{lines >> 2, plane}; return z0 + t.offset(l) + e * t.stride(); }
    if (kind == 3) { const sim::TileLines<3> t{lines >> 3, plane}; return z0 + t.offset(l) + e * t.stride(); }
    const sim::GridLines g = grid();
    return z0 + g.offset(l) + e * g.stride();
}
// kind (0: columns of a grid, 1: its rows, 2 and 3: tiles of 4 and 8 lines a plane), length, lines, threads
int main(int argc, char **argv) {
    kind = std::atoi(argv[1]);
    n = std::atoi(argv[2]);
    lines = std::atoi(argv[3]);
    const int threads = std::atoi(argv[4]);
    const sim::FftPlan p = sim::fft_plan(n, kind < 2 ? 8 : 24);
    sim::fft_plans[0] = p;
    int product = 1;
    for (int i = 0; i < p.stages; ++i) product *= p.at[i].r;
    if (product != n) { std::puts("plan"); return 3; }
    z0 = (n + 15) / 16 * 16;
    plane = kind == 2 ? 4 * n : kind == 3 ? 8 * n : 0;
    room = z0 + (kind == 1 ? lines * (n | 1) : lines * n);
    if (room > kRoom) { std::puts("room"); return 3; }
    for (int i = 0; i < n; ++i)
        sim::fft_sm[i] = float2((float)std::cos(2 * M_PI * i / n), (float)-std::sin(2 * M_PI * i / n));
    std::vector<double> xr(lines * n), xi(lines * n);
    unsigned state = 12345u + n;
    auto draw = [&] { state = state * 1664525u + 1013904223u; return (float)(state >> 8) / 8388608.f - 1.f; };
    double worst = 0;
    for (int dir = 0; dir < 2; ++dir) {
        in_time = dir;
        for (int l = 0; l < lines; ++l)
            for (int e = 0; e < n; ++e) {
                const float a = draw(), b = draw();
                xr[l * n + e] = a;
                xi[l * n + e] = b;
                sim::fft_sm[place(l, e)] = float2(a, b);
            }
        ++phase;
        run_block(threads, transform);
        std::vector<int> order(n);
        for (int e = 0; e < n; ++e) order[e] = sim::fft_index_at(p, e);
        for (int l = 0; l < lines; l += std::max(1, lines / 3))
            for (int e = 0; e < n; ++e) {
                double ar = 0, ai = 0;
                const int k = dir ? e : order[e];
                for (int j = 0; j < n; ++j) {
                    const int src = dir ? order[j] : j;
                    const double w = -2 * M_PI * ((long long)k * src % n) / n;
                    ar += xr[l * n + j] * std::cos(w) - xi[l * n + j] * std::sin(w);
                    ai += xr[l * n + j] * std::sin(w) + xi[l * n + j] * std::cos(w);
                }
                const float2 &v = sim::fft_sm[place(l, e)];
                worst = std::max(worst, std::hypot(v.x - ar, v.y - ai) / std::sqrt((double)n));
            }
    }
    std::printf("races %d outside %d error %.3g\n", races, outside, worst);
    return 0;
}
"""


@pytest.fixture(scope="module")
def harness(tmp_path_factory):
    d = tmp_path_factory.mktemp("simfft")
    shutil.copy(os.path.join(CSRC, "simfft.cuh"), d)
    (d / "common.cuh").write_text(SHIM)
    (d / "main.cpp").write_text(MAIN)
    subprocess.run(["g++", "-std=c++17", "-O1", "-w", "-ffp-contract=off", "-o", str(d / "main"), str(d / "main.cpp")], check=True)
    return str(d / "main")


# columns and rows of a cluster's block: small radices, primes by direct sums with one, two and four outputs a thread,
# in one pass over the butterflies and in several whose last leaves threads without work; tiles: every radix, primes
# beyond 23, four lines and eight, one plane and two
@pytest.mark.parametrize("kind, n, lines, threads", [
    (0, 43, 3, 256), (0, 43, 6, 256), (1, 47, 6, 256), (0, 113, 8, 512), (1, 109, 15, 512), (1, 113, 57, 512),
    (0, 62, 10, 512), (1, 79, 31, 512), (0, 60, 17, 256), (1, 64, 8, 256), (0, 45, 7, 256), (1, 98, 4, 256), (0, 5, 1, 256),
    (0, 33, 40, 256), (1, 22, 200, 512),
    (2, 552, 4, 256), (3, 552, 16, 256), (3, 288, 8, 256), (2, 259, 8, 256), (3, 266, 16, 256), (2, 1147, 4, 256),
    (3, 899, 8, 256), (2, 1001, 4, 256), (3, 2210, 8, 256), (2, 1024, 8, 256), (3, 900, 8, 256), (2, 1332, 8, 256)])
def test_transforms_without_races(harness, kind, n, lines, threads):
    r = subprocess.run([harness, str(kind), str(n), str(lines), str(threads)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    f = r.stdout.split()
    assert f[1] == "0" and f[3] == "0", r.stdout
    assert float(f[5]) < 1e-5, r.stdout
