"""Which arrays the state transfer's kernel takes, and the device it is launched under, with another device
current than the solver's: csrc/device_scope.cuh against a fake of the runtime calls it makes (two
devices, no GPU)."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r'''
#include <cstdio>
#include <map>
#include "device_scope.cuh"

static int current = 0;
struct Range { cudaPointerAttributes a; uintptr_t size; };
static std::map<uintptr_t, Range> memory;
extern "C" {
cudaError_t cudaGetDevice(int *d) { *d = current; return cudaSuccess; }
cudaError_t cudaSetDevice(int d) { current = d; return d < 2 ? cudaSuccess : cudaErrorInvalidDevice; }
cudaError_t cudaGetLastError(void) { return cudaSuccess; }
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes *a, const void *p)
{
    const uintptr_t v = reinterpret_cast<uintptr_t>(p);
    auto it = memory.upper_bound(v);
    if (it == memory.begin()) return cudaErrorInvalidValue;
    --it;
    if (v - it->first >= it->second.size) return cudaErrorInvalidValue;
    *a = it->second.a;
    if (a->devicePointer) a->devicePointer = const_cast<void *>(p);
    return cudaSuccess;
}
}
#define EXPECT(c) do { if (!(c)) { std::printf("FAILED %s (line %d)\n", #c, __LINE__); return 1; } } while (0)

int main()
{
    auto add = [&](uintptr_t v, uintptr_t size, cudaMemoryType t, int device, bool mapped) {
        cudaPointerAttributes a{};
        a.type = t;
        a.device = device;
        a.devicePointer = mapped ? reinterpret_cast<void *>(v) : nullptr;
        memory[v] = Range{a, size};
    };
    const size_t n = 9 * 256;
    add(0x10000, 4 * n, cudaMemoryTypeDevice, 0, true);
    add(0x20000, 4 * n, cudaMemoryTypeDevice, 1, true);
    add(0x30000, 4 * n, cudaMemoryTypeManaged, 0, true);
    add(0x40000, 4 * n, cudaMemoryTypeHost, 0, true);
    add(0x50000, 4 * n, cudaMemoryTypeUnregistered, 0, false);
    add(0x60000, 4 * n + 4, cudaMemoryTypeDevice, 0, true);
    auto reach = [&](uintptr_t v, int solver, size_t count) {
        return crb200::kernelReachable(reinterpret_cast<void *>(v), count, solver);
    };
    for (int solver = 0; solver < 2; ++solver)
        for (current = 0; current < 2; ++current)
        {
            const int was = current;
            EXPECT(reach(0x10000, solver, n) == (solver == 0));
            EXPECT(reach(0x20000, solver, n) == (solver == 1));
            EXPECT(reach(0x30000, solver, n));
            EXPECT(reach(0x40000, solver, n));
            EXPECT(!reach(0x50000, solver, n));
            EXPECT(!reach(0x60002, solver, n)); // odd address
            EXPECT(!reach(0x70000, solver, n)); // unknown
            EXPECT(!reach(0x30000, solver, n + 1) && !reach(0x40004, solver, n)); // ends early
            EXPECT(reach(0x30000, solver, 1));
            {
                const crb200::DeviceScope scope(solver);
                EXPECT(current == solver);
            }
            EXPECT(current == was);
        }
    std::printf("ok\n");
    return 0;
}
'''


def test_state_transfer_with_another_device_current(tmp_path):
    src, exe = tmp_path / "device_scope.cpp", tmp_path / "device_scope"
    src.write_text(PROGRAM)
    cmd = ["g++", "-std=c++17", "-Wall", "-Werror", f"-I{ROOT}/cressim-mpm_b200/csrc", "-I/usr/local/cuda/include",
           str(src), "-o", str(exe)]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-3000:]
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout
