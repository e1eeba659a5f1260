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
