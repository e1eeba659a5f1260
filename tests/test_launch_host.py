"""Host side of the launches (csrc/ov_host.h) on a fake CUDA runtime: two
devices of different size in one process."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "odevec_b200", "csrc")

FAKE_DEVICES = r"""
#include "ov_host.h"
#include <cstdio>
#include <map>
static int g_dev = 0, g_queries = 0;
static std::map<int, int> g_limit; /* device -> the kernel's shared-memory limit */
extern "C" cudaError_t cudaGetDevice(int* d) { *d = g_dev; return cudaSuccess; }
extern "C" cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int dev)
{
    *v = dev == 0 ? 148 : 100;
    return cudaSuccess;
}
extern "C" cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int v)
{
    g_limit[g_dev] = v;
    return cudaSuccess;
}
extern "C" cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int* n, const void*, int block, size_t)
{
    ++g_queries;
    *n = 512 / block;
    return cudaSuccess;
}
#define CHECK(x) do { if (!(x)) { std::printf("line %d: %s\n", __LINE__, #x); return 1; } } while (0)
static int launch(ov::Residency& r, int block, size_t smem)
{
    const char kern = 0;
    int grid = -1;
    if (ov::allow_smem(&kern, smem) != cudaSuccess || ov::resident_blocks(r, &kern, block, smem, &grid) != cudaSuccess)
        return -1;
    /* the launch itself fails without the limit on this device */
    return smem > 48 * 1024 && (size_t)g_limit[g_dev] < smem ? -2 : grid;
}
"""


def _run(tmp_path, source):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    inc = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(nvcc))), "include")
    if not os.path.exists(os.path.join(inc, "cuda_runtime_api.h")):
        pytest.skip("no CUDA headers")
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(source)
    subprocess.run(["g++", "-std=c++17", "-Wall", "-I" + inc, "-I" + CSRC, "-o", str(exe), str(src)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout + r.stderr


def test_launch_on_two_devices(tmp_path):
    """Each device gets the kernel's shared-memory limit and a grid of its own
    size; a reset device gets the limit again; occupancy is asked once per
    device and block size."""
    _run(tmp_path, FAKE_DEVICES + r"""
int main()
{
    static ov::Residency r;
    CHECK(launch(r, 256, 200 * 1024) == 148 * 2);
    g_dev = 1;
    CHECK(launch(r, 256, 200 * 1024) == 100 * 2);
    g_limit.clear(); /* both devices reset */
    CHECK(launch(r, 256, 200 * 1024) == 100 * 2);
    g_dev = 0;
    CHECK(launch(r, 256, 200 * 1024) == 148 * 2);
    CHECK(g_queries == 2);
    CHECK(launch(r, 128, 0) == 148 * 4);
    CHECK(g_queries == 3);
    g_dev = ov::Residency::DEVICES; /* beyond the kept ones */
    CHECK(launch(r, 128, 0) == 100 * 4 && launch(r, 128, 0) == 100 * 4);
    CHECK(g_queries == 5);
    return 0;
}
""")


FAKE_MEMORY = r"""
#include "rate_tables.hpp"
#include <cstdio>
#include <cstdlib>
#include <map>
static size_t g_room = 0;
static bool g_capturing = false;
static std::map<void*, size_t> g_live;
extern "C" cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus* s)
{
    *s = g_capturing ? cudaStreamCaptureStatusActive : cudaStreamCaptureStatusNone;
    return cudaSuccess;
}
extern "C" cudaError_t cudaGetLastError() { return cudaSuccess; }
extern "C" cudaError_t cudaThreadExchangeStreamCaptureMode(cudaStreamCaptureMode*) { return cudaSuccess; }
extern "C" cudaError_t cudaMemGetInfo(size_t* f, size_t* t) { *f = g_room; *t = g_room; return cudaSuccess; }
extern "C" cudaError_t cudaMalloc(void** p, size_t n)
{
    if (g_capturing || n > g_room)
        return cudaErrorMemoryAllocation;
    *p = std::malloc(1);
    g_live[*p] = n;
    g_room -= n;
    return cudaSuccess;
}
extern "C" cudaError_t cudaFree(void* p)
{
    if (g_live.count(p) != 1)
        std::abort();
    g_room += g_live[p];
    g_live.erase(p);
    std::free(p);
    return cudaSuccess;
}
static size_t live() { size_t n = 0; for (auto& e : g_live) n += e.second; return n; }
#define CHECK(x) do { if (!(x)) { std::printf("line %d: %s\n", __LINE__, #x); return 1; } } while (0)
"""


def test_rate_tables_memory(tmp_path):
    """A solver whose cell count grows holds one table; a table in a graph stays
    where it is; none is taken where it would leave less than half of the free
    memory; what no graph holds can be given back."""
    _run(tmp_path, FAKE_MEMORY + r"""
int main()
{
    const int64_t nrea = 38, B = 8 * nrea;
    g_room = 12000 * B; /* half of what the table of at most 2,248 cells leaves holds twice as much */
    ov::RateTables r = {};
    double* a = r.get(1000, nrea, 0);
    CHECK(a && live() == (size_t)(1000 * B));
    CHECK(r.get(700, nrea, 0) == a && r.get(1000, nrea, 0) == a);
    for (int64_t n = 1001; n < 2000; ++n) { /* one table, at most an eighth too large */
        CHECK(r.get(n, nrea, 0) && live() >= (size_t)(n * B) && live() <= (size_t)((n + n / 8) * B));
    }
    g_capturing = true;
    double* g = r.get(1500, nrea, 0); /* now in a graph */
    const size_t held = live();
    CHECK(g && r.get(9000, nrea, 0) == nullptr && live() == held);
    g_capturing = false;
    CHECK(r.get(1500, nrea, 0) == g && !r.drop());
    double* b = r.get(3000, nrea, 0);
    CHECK(b && b != g && live() >= 3 * held); /* at least twice the one before */
    CHECK(r.drop() && live() == held && !r.drop());
    CHECK(r.get(9000, nrea, 0) == nullptr && live() == held); /* more than half of what is free */
    CHECK(r.get(3000, nrea, 0) && r.get(1500, nrea, 0));
    r.close();
    CHECK(live() == 0 && r.n == 0 && r.get(1000, nrea, 0));
    r.close();
    return 0;
}
""")


def test_rate_tables_give_way(tmp_path):
    """A buffer that a solve needs takes the place of the newest table where there
    is no room for both, but not of a table that a graph may hold."""
    _run(tmp_path, FAKE_MEMORY + r"""
int main()
{
    const int64_t nrea = 38, B = 8 * nrea;
    g_room = 2000 * B;
    ov::RateTables r = {};
    double* p = nullptr;
    CHECK(r.get(1000, nrea, 0) && r.alloc(&p, 900 * B) == cudaSuccess && r.n == 1);
    cudaFree(p);
    CHECK(r.alloc(&p, 1500 * B) == cudaSuccess && r.n == 0 && live() == (size_t)(1500 * B));
    CHECK(r.get(1000, nrea, 0) == nullptr); /* the solve then goes without */
    cudaFree(p);
    CHECK(r.get(1000, nrea, 0));
    g_capturing = true;
    CHECK(r.get(1000, nrea, 0));
    g_capturing = false;
    CHECK(r.alloc(&p, 1500 * B) == cudaErrorMemoryAllocation && r.n == 1);
    r.close();
    return 0;
}
""")


def test_launch_loads_one_kernel():
    """The launcher hands a solve of few cells to the other shape's kernel before
    it asks the runtime anything about its own, which would load it."""
    text = open(os.path.join(CSRC, "bdf_kernel.cuh")).read()
    body = text[text.index("cudaError_t launch(const LaunchArgs& a, int block, int grid"):]
    body = body[:body.index("kern<<<")]
    other = body.index("return launch<Net, G, LUT, SPREAD_STAGE>")
    for question in ("allow_smem(", "resident_blocks("):
        assert body.count(question) == 1 and body.index(question) > other
