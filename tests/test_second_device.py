"""The launches that need a kernel attribute or a device's size, on a second
device of the same process. The library's launch code is linked with a CUDA
runtime of two made-up devices, so this runs without a GPU: a launch with
dynamic shared memory or with a cluster of more than 8 CTAs passes only where
its kernel was given the attribute on the device it runs on."""
import os
import subprocess

import pytest

PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "dirty-gen_b200")
OBJECTS = [os.path.join(PKG, "_build", o + ".o") for o in ("sheet_window", "sheet_grid", "closure_mma")]
RUNTIME = r"""
#include <cuda_runtime_api.h>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <set>
#include <utility>

// Two devices: the first of 148 SMs, the second of 60 that holds crews of up to 4.
int device = 0, refused = 0;
const void* kernel = nullptr;  // of the last launch
int fail_attribute = -1;  // the device that refuses shared memory
unsigned grid = 0, cluster = 0;
static const int SMS[2] = {148, 60}, CREW[2] = {16, 4};
static std::map<std::pair<int, const void*>, int> smem;
static std::set<std::pair<int, const void*>> large;
static cudaError_t last = cudaSuccess;

extern "C" {
void** __cudaRegisterFatBinary(void*) { static void* h; return &h; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char*, char*, const char*, int, uint3*, uint3*, dim3*, dim3*, int*) {}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
char __cudaInitModule(void**) { return 0; }
cudaError_t __cudaPopCallConfiguration(dim3*, dim3*, size_t*, void*) { return cudaErrorUnknown; }
unsigned __cudaPushCallConfiguration(dim3, dim3, size_t, cudaStream_t) { return 1; }
cudaError_t cudaLaunchKernel(const void*, dim3, dim3, void**, size_t, cudaStream_t) { return cudaErrorUnknown; }
cudaError_t cudaGetDevice(int* d) { *d = device; return cudaSuccess; }
cudaError_t cudaGetLastError() { return std::exchange(last, cudaSuccess); }
const char* cudaGetErrorString(cudaError_t) { return "error"; }
cudaError_t cudaMalloc(void** p, size_t n) { *p = malloc(n); return cudaSuccess; }
cudaError_t cudaMemset(void* p, int v, size_t n) { memset(p, v, n); return cudaSuccess; }
cudaError_t cudaMemsetAsync(void*, int, size_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void*, const void*, size_t, cudaMemcpyKind, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr a, int d) {
    if (a != cudaDevAttrMultiProcessorCount || d < 0 || d > 1) return cudaErrorInvalidValue;
    *v = SMS[d];
    return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void* f, cudaFuncAttribute a, int v) {
    if (a == cudaFuncAttributeMaxDynamicSharedMemorySize) {
        if (device == fail_attribute) return last = cudaErrorInvalidValue;
        smem[{device, f}] = v;
    }
    if (a == cudaFuncAttributeNonPortableClusterSizeAllowed && v) large.insert({device, f});
    return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveClusters(int* n, const void*, const cudaLaunchConfig_t* c) {
    *n = c->attrs[0].val.clusterDim.x <= (unsigned)CREW[device];
    return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void*, int, size_t, unsigned) {
    *n = 2;
    return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int* n, const void*, int, size_t) {
    *n = 2;
    return cudaSuccess;
}
cudaError_t cudaGetDriverEntryPoint(const char*, void**, unsigned long long, cudaDriverEntryPointQueryResult*) {
    return cudaErrorNotSupported;
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void**) {
    kernel = f;
    grid = c->gridDim.x;
    cluster = 1;
    for (unsigned k = 0; k < c->numAttrs; ++k)
        if (c->attrs[k].id == cudaLaunchAttributeClusterDimension) cluster = c->attrs[k].val.clusterDim.x;
    const auto it = smem.find({device, f});
    const bool room = c->dynamicSmemBytes == 0 || (it != smem.end() && (size_t)it->second >= c->dynamicSmemBytes);
    if (!room || cluster > (unsigned)CREW[device] || (cluster > 8 && !large.count({device, f}))) {
        ++refused;
        return last = cudaErrorInvalidValue;
    }
    return cudaSuccess;
}
}
"""
PROGRAM = r"""
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include "closure.cuh"
#include "sheet_grid.cuh"
#include "sheet_window.cuh"

extern int device, refused, fail_attribute;
extern const void* kernel;
extern unsigned grid, cluster;

namespace silt {
thread_local unsigned long long t_kernel_launches = 0;
bool kernel_timing_on() { return false; }
void kernel_timing_begin(cudaStream_t) {}
void kernel_timing_end(cudaStream_t, const void*) {}
}  // namespace silt

using namespace silt;

int main(int argc, char** argv) {
    if (argc > 1) fail_attribute = atoi(argv[1]);
    static SweepState sweep;
    static uint16_t x[64];
    static float f[64];
    for (int d : {0, 1, 0, 1}) {
        device = d;
        refused = 0;
        int failed = 0;
        auto ran = [&](cudaError_t e) { failed += e != cudaSuccess; };
        for (int res : {64, 200, 512}) {
            ran(window::launch_window_step(nullptr, 1, res, nullptr));
            ran(window::launch_window_step_list(nullptr, 1, res, nullptr));
        }
        const unsigned crew = cluster;
        ForceLaunch F;
        memset(&F, 0, sizeof F);
        F.tf.sweep = &sweep;
        ran(launch_force(F, 64, 2, nullptr));
        // 32-bit places up to 46340 cells a side, a kernel of its own above.
        const void* const near = kernel;
        ran(launch_force(F, 46340, 2, nullptr));
        failed += kernel != near;
        ran(launch_force(F, 46341, 2, nullptr));
        const int far = kernel != near;
        F.lay[0].sweep = 1;
        ran(launch_force(F, 64, 2, nullptr));
        const unsigned coop = grid;
        ran(launch_batch_force(nullptr, 1, nullptr, nullptr, nullptr, &sweep, false, nullptr));
        const unsigned batch = grid;
        ran(launch_batch_force(nullptr, 1, nullptr, nullptr, nullptr, nullptr, true, nullptr));
        TransportLaunch T;
        memset(&T, 0, sizeof T);
        ran(launch_transport(T, 64, 2, nullptr));
        ran(launch_batch_transport(nullptr, nullptr, nullptr, nullptr, nullptr));
        ran(closure::conv3x3(x, x, f, nullptr, x, nullptr, 64, 32, 32, 32, 32, 1, nullptr));
        const unsigned conv = grid;
        ran(closure::conv3x3_wgrad(x, x, f, f, 64, 32, 32, 32, 32, nullptr));
        printf("%d %d %d %u %u %u %u %d\n", d, failed, refused, crew, coop, batch, conv, far);
    }
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    subprocess.check_call(["make", "-s", "-j4", "-C", PKG] + OBJECTS)
    d = tmp_path_factory.mktemp("devices")
    (d / "runtime.cpp").write_text(RUNTIME)
    (d / "devices.cu").write_text(PROGRAM)
    subprocess.check_call(["nvcc", "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-cudart", "none", "-I",
                           os.path.join(PKG, "csrc"), str(d / "runtime.cpp"), str(d / "devices.cu")] + OBJECTS +
                          ["-o", str(d / "devices")])
    return str(d / "devices")


def rows(program, *args):
    out = subprocess.check_output([program, *args], text=True)
    return [tuple(map(int, ln.split())) for ln in out.splitlines()]


def test_every_launch_on_each_device(program):
    """No launch is refused, and crews and grids are each device's own."""
    first, second = (0, 0, 0, 16, 148 * 2, 148 * 2, 512, 1), (1, 0, 0, 4, 60 * 2, 60 * 2, 4 * 60, 1)
    assert rows(program) == [first, second, first, second]


def test_a_device_that_refuses_shared_memory_says_so(program):
    """Every call there returns an error and launches nothing; the other device is not touched by it."""
    got = rows(program, "1")
    assert [r[0] for r in got] == [0, 1, 0, 1]
    assert all(r[1:3] == (0, 0) for r in got if r[0] == 0)
    assert all(r[1:3] == (16, 0) for r in got if r[0] == 1)
