"""A failing call leaves nothing running in memory that its caller takes back.

The RF simulation and the DTFT are compiled against a stand-in for the CUDA
runtime that records what is queued on the stream and answers one call, the
first, the second and so on, with an error.  Whatever fails: the entry point
reports it, and has waited for the stream since the last work that it queued
there, both in a caller's workspace and in memory of its own, which it frees."""
import os
import subprocess

import pytest

from waveforminversionust_b200.build import CSRC, ROOT, nvcc

RUNTIME = r"""
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <vector>
#include <cuda_runtime_api.h>
#include "wust_b200.h"

static int calls, fail_at, queued, pending, freed, taken;
static cudaError_t last;
static cudaStream_t const kStream = (cudaStream_t)0x77;
static void wrong(const char *what) { std::printf("%s\n", what); std::exit(1); }
// work on the stream: accepted, or refused where it is this call's turn
static cudaError_t work(cudaStream_t st) {
    if (st != kStream) wrong("another stream");
    if (++calls == fail_at) return last = cudaErrorLaunchOutOfResources;
    ++queued;
    pending = 1;
    return cudaSuccess;
}
extern "C" {
struct Config { dim3 g, b; size_t smem; cudaStream_t st; };
static Config config;
void **__cudaRegisterFatBinary(void *) { static void *h; return &h; }
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterFunction(void **, const char *, char *, const char *, int, uint3 *, uint3 *, dim3 *, dim3 *, int *) {}
void __cudaRegisterVar(void **, char *, char *, const char *, int, size_t, int, int) {}
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t smem, cudaStream_t st) {
    config = Config{g, b, smem, st};
    return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3 *g, dim3 *b, size_t *smem, void *st) {
    *g = config.g;
    *b = config.b;
    *smem = config.smem;
    *(cudaStream_t *)st = config.st;
    return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void *, dim3, dim3, void **, size_t, cudaStream_t st) { return work(st); }
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t *c, const void *, void **) { return work(c->stream); }
cudaError_t cudaMemcpyAsync(void *, const void *, size_t, cudaMemcpyKind, cudaStream_t st) { return work(st); }
cudaError_t cudaMemsetAsync(void *, int, size_t, cudaStream_t st) { return work(st); }
cudaError_t cudaFuncSetAttribute(const void *, cudaFuncAttribute, int) {
    return ++calls == fail_at ? (last = cudaErrorInvalidValue) : cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t st) {
    if (st != kStream) wrong("another stream");
    pending = 0;
    return ++calls == fail_at ? (last = cudaErrorUnknown) : cudaSuccess;
}
cudaError_t cudaMallocAsync(void **p, size_t, cudaStream_t) {
    *p = (void *)0x200000;
    if (++calls == fail_at) return last = cudaErrorMemoryAllocation;
    ++taken;
    return cudaSuccess;
}
cudaError_t cudaFreeAsync(void *p, cudaStream_t) {
    if (p != (void *)0x200000) wrong("freed what is not its own");
    ++freed;
    return cudaSuccess;
}
cudaError_t cudaMalloc(void **p, size_t) {
    *p = (void *)0x600000;
    if (++calls == fail_at) return last = cudaErrorMemoryAllocation;
    ++taken;
    return cudaSuccess;
}
cudaError_t cudaFree(void *p) {
    if (p != (void *)0x600000 || pending) wrong("freed what is not its own, or in use");
    ++freed;
    return cudaSuccess;
}
cudaError_t cudaPeekAtLastError() { return last; }
cudaError_t cudaGetLastError() { const cudaError_t e = last; last = cudaSuccess; return e; }
const char *cudaGetErrorString(cudaError_t) { return "made up"; }
}

static std::vector<double> c, source, t, f;
static std::vector<int> tx, rx;
static int ny, nx, nt = 6, q, batch;
static int simulate(void *ws, size_t bytes) {
    return wust_simulate_ws(c.data(), ny, nx, 1e-3, 1e-3, 1e-7, nt, source.data(), tx.data(), (int)tx.size(), rx.data(),
                            (int)rx.size(), 4, 1600, 1000, q, batch, (float *)0x300000, ws, bytes, kStream);
}
static int dtft(void *ws, size_t bytes) {
    return wust_dtft_ws(t.data(), (int)t.size(), f.data(), (int)f.size(), (void *)0x300000, 0, 3, 5, (uint8_t *)0x400000,
                        (wust_c64 *)0x500000, ws, bytes, kStream);
}
static void every_failure(const char *name, int (*call)(void *, size_t), size_t bytes) {
    for (int own = 0; own < 2; ++own) {
        int failed = 0;
        for (fail_at = 1;; ++fail_at) {
            calls = queued = pending = freed = taken = 0;
            last = cudaSuccess;
            const int rc = own ? call(nullptr, 0) : call((void *)0x100000, bytes);
            const bool hit = calls >= fail_at;
            if (hit == (rc == WUST_OK)) { std::printf("%s, call %d: status %d\n", name, fail_at, rc); std::exit(1); }
            if (pending) { std::printf("%s, call %d failed: returned with work on the stream\n", name, fail_at); std::exit(1); }
            if (freed != taken) { std::printf("%s, call %d: memory kept\n", name, fail_at); std::exit(1); }
            if (!hit) break;
            ++failed;
        }
        std::printf("%s %d: %d failures, %d pieces of work\n", name, own, failed, queued);
        if (failed < 3) wrong("nothing failed");
    }
}
int main() {
    // a cluster's grid, tiles, their records decimated, and fields that a pool does not hold
    const int grids[][4] = {{11, 13, 1, 1}, {240, 232, 1, 1}, {240, 232, 3, 1}, {512, 504, 1, 0}};
    for (const auto &g : grids) {
        ny = g[0];
        nx = g[1];
        q = g[2];
        batch = g[3];
        c.assign((size_t)ny * nx, 1500.0);
        source.assign(nt, 1.0);
        tx = {3, 8};
        for (int i = 0; !batch && i < 10; ++i) tx.push_back(20 + i);
        rx = {5, 9, 70};
        const size_t bytes = wust_simulate_workspace_bytes(ny, nx, 4, (int)tx.size(), (int)rx.size(), nt, q, batch);
        if (!bytes) wrong("not the path meant");
        every_failure("simulate", simulate, bytes);
    }
    f = {1e5, 2e5};
    for (int uneven = 0; uneven < 2; ++uneven) {
        t.assign(40, 0);
        for (int i = 0; i < 40; ++i) t[i] = 1e-7 * (i + (uneven && i == 7 ? 1e-7 : 0));
        every_failure(uneven ? "dtft, uneven" : "dtft", dtft, wust_dtft_workspace_bytes(40, 2));
    }
    return 0;
}
"""


def test_errors_leave_no_work_behind(tmp_path):
    flags = ["-std=c++17", "-O1", "-I", os.path.join(ROOT, "include")]
    (tmp_path / "main.cpp").write_text(RUNTIME)
    names = ["api", "simulate", "prepare"]
    # the host's side is what runs: device code as far as PTX
    builds = [subprocess.Popen([nvcc(), *flags, "--expt-relaxed-constexpr", "-gencode", "arch=compute_100a,code=compute_100a",
                                "-Xcompiler", "-fPIC", "-c", os.path.join(CSRC, n + ".cu"), "-o", str(tmp_path / (n + ".o"))])
              for n in names]
    builds.append(subprocess.Popen([nvcc(), *flags, "-c", str(tmp_path / "main.cpp"), "-o", str(tmp_path / "main.o")]))
    assert all(b.wait() == 0 for b in builds)
    exe = str(tmp_path / "main")
    # entry points of the other files are not called
    subprocess.run(["g++", "-o", exe, *[str(tmp_path / (n + ".o")) for n in ["main", *names]],
                    "-Wl,--unresolved-symbols=ignore-all"], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
