"""Kernels with more than 48 KB of shared memory are granted it once on every device."""
import ctypes

from host_kernels import compile_host, section

TAIL = r"""
#include <thread>
void kernel_a() {}
void kernel_b() {}
extern "C" void launch(int dev, int which) {
  std::thread([&] {
    device = dev;
    if (which) allow_smem<kernel_b>(70000);
    else allow_smem<kernel_a>(60000);
  }).join();
}
extern "C" int granted(int dev, int which) { return grants[dev][which ? (void*)kernel_b : (void*)kernel_a]; }
"""
FAKE = r"""
#include <atomic>
#include <map>
thread_local int device = 0;
std::map<void*, int> grants[80];
enum { cudaFuncAttributeMaxDynamicSharedMemorySize };
void cudaGetDevice(int* d) { *d = device; }
template <typename F> void cudaFuncSetAttribute(F f, int, int bytes) { if (bytes > 48 << 10) ++grants[device][(void*)f]; }
"""


def test_every_device_once():
    lib = compile_host([FAKE, section("kernels.cuh", "template <auto Kernel>", "// an integer constant")], TAIL)
    for dev in (0, 1, 0, 3, 1, 0):
        for which in (0, 1):
            lib.launch(dev, which)
    assert [[lib.granted(d, k) for k in (0, 1)] for d in range(4)] == [[1, 1], [1, 1], [0, 0], [1, 1]]
