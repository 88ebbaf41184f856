"""pf_limits.h against a CUDA runtime of its own that keeps each kernel's
limit per device: a limit never falls under a size that was asked for before,
whatever the order and number of sizes, kernels, devices and threads; what is
kept is asked once, what was pushed out again; too large a size is refused."""
import subprocess

import pytest

from pixelforge_gb300.build import CSRC, _cuda_home

SOURCE = r"""
#include "pf_limits.h"
#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <thread>
#include <vector>
#define CHECK(c) do { if (!(c)) { std::printf("line %d: %s\n", __LINE__, #c); std::exit(1); } } while (0)
enum { DEVICES = 8, KERNELS = 18, OPTIN = 232448, STATIC = 48 };
static thread_local int device = 0;
static std::atomic<int> limit[DEVICES][KERNELS];
static std::atomic<int> calls{ 0 };
static int at(const void *k) { return (int)((const char *)k - (const char *)&limit); }
static const void *kernel(int k) { return (const char *)&limit + k; }
extern "C" {
cudaError_t cudaGetDevice(int *d) { *d = device; return cudaSuccess; }
cudaError_t cudaFuncGetAttributes(cudaFuncAttributes *a, const void *k)
{
    calls++;
    *a = cudaFuncAttributes{};
    a->sharedSizeBytes = STATIC;
    a->maxDynamicSharedSizeBytes = limit[device][at(k)];
    return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void *k, cudaFuncAttribute a, int v)
{
    if (a != cudaFuncAttributeMaxDynamicSharedMemorySize) return cudaSuccess;
    if (v < 0 || v > OPTIN - STATIC) return cudaErrorInvalidValue;
    limit[device][at(k)] = v;
    return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int *fit, const void *k, int block, size_t smem)
{
    if ((int)smem > limit[device][at(k)]) return cudaErrorInvalidValue;
    *fit = 1 + (int)(smem / 1000) + block + 7 * at(k);
    return cudaSuccess;
}
}
// asks, and checks what a launch of that size needs
static void ask(int d, int k, size_t smem)
{
    device = d;
    int fit = 0;
    CHECK(pfd_ctas_per_sm(kernel(k), 128, smem, k % 2 != 0, fit) == cudaSuccess);
    CHECK(fit == 1 + (int)(smem / 1000) + 128 + 7 * k);
    CHECK(limit[d][k] >= (int)smem);
}
int main()
{
    for (auto &d : limit) for (auto &l : d) l = 49152;
    // one device's sizes are asked once each
    for (int pass = 0; pass < 3; pass++) {
        for (int k = 0; k < 4; k++) for (int i = 0; i < 10; i++) ask(0, k, 256u << i);
        CHECK(calls == 40);
    }
    int big = 0;
    CHECK(pfd_ctas_per_sm(kernel(0), 128, OPTIN, false, big) == cudaErrorInvalidValue && limit[0][0] >= 256 << 9);
    // many more than are kept, on several devices, the large ones first: no limit falls
    std::vector<size_t> most(DEVICES * KERNELS, 0);
    for (int i = 12; i >= 0; i--)
        for (int d = 0; d < DEVICES; d++)
            for (int k = 0; k < KERNELS; k++) {
                const size_t s = 30000 + 16000u * (size_t)i + 16u * (size_t)k;
                ask(d, k, s);
                size_t &m = most[(size_t)(d * KERNELS + k)];
                m = s > m ? s : m;
                CHECK(limit[d][k] >= (int)m);
            }
    // what was asked last is kept, however much was asked before
    int before = calls;
    for (int k = 0; k < KERNELS; k++) ask(DEVICES - 1, k, 30000 + 16u * (size_t)k);
    CHECK(calls == before);
    // threads with sizes of their own: each finds its limit after its call, at any later time
    std::vector<std::thread> ts;
    for (int t = 0; t < 4; t++)
        ts.emplace_back([t] {
            for (int i = 0; i < 3000; i++) {
                const int k = i % KERNELS, d = i % 2;
                const size_t s = 50000 + 16u * (size_t)((i * 7919 + t * 104729) % 10000);
                ask(d, k, s);
                std::this_thread::yield();
                CHECK(limit[d][k] >= (int)s);
            }
        });
    for (auto &t : ts) t.join();
    std::puts("ok");
}
"""


def test_limits_are_never_lowered(tmp_path):
    src, exe = tmp_path / "limits.cpp", tmp_path / "limits"
    src.write_text(SOURCE)
    try:
        cuda = _cuda_home()
    except RuntimeError as e:
        pytest.skip(str(e))
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", f"-I{CSRC}", f"-I{cuda / 'include'}", str(src), "-o", str(exe)],
                   check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and r.stdout == "ok\n", r.stdout
