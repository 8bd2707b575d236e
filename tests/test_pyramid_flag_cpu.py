"""The record that the count pyramid is zero (Builder::pyr_zero_), on the CPU: builder.cpp linked against a stand-in of
the CUDA runtime whose cudaMalloc returns the address that was freed last, as the real one may for a larger size."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "octree-cuda_gb300", "csrc")
CUDA_INC = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")

PROGRAM = r"""
#include <cstdlib>
#define private public
#include "builder.h"
static void* freed = nullptr;
static uintptr_t next = 1 << 20;
extern "C" cudaError_t cudaMalloc(void** p, size_t) {
    *p = freed ? freed : reinterpret_cast<void*>(next += 256);
    freed = nullptr;
    return cudaSuccess;
}
extern "C" cudaError_t cudaFree(void* p) { freed = p; return cudaSuccess; }
extern "C" cudaError_t cudaMallocHost(void** p, size_t n) { *p = std::calloc(1, n); return cudaSuccess; }
extern "C" cudaError_t cudaFreeHost(void* p) { std::free(p); return cudaSuccess; }
extern "C" cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) { *v = 152; return cudaSuccess; }
extern "C" const char* cudaGetErrorString(cudaError_t) { return ""; }

int main() {
    using namespace oc;
    BuildConfig c;
    c.n = 1000;
    c.stride = 15;
    c.chunk_grid = 64;
    c.threshold = 100;
    c.output_factor = 2.2f;
    c.sub_grid = 128;
    for (int a = 0; a < 3; ++a) c.bb_max[a] = 1.0;
    const uint8_t cloud[16] = {};
    Builder b(c, cloud, 0);
    const void* old = b.pyr_.p;
    b.pyr_zero_ = true;            // as a build leaves it
    b.reconfigure(c, cloud);
    if (!b.pyr_zero_) return 1;    // the same buffers
    c.chunk_grid = 128;
    b.reconfigure(c, cloud);
    if (b.pyr_.p != old) return 2; // the case in question
    return b.pyr_zero_ ? 3 : 0;    // a larger allocation holds garbage
}
"""


@pytest.mark.skipif(not shutil.which("g++") or not shutil.which("nm") or not os.path.exists(CUDA_INC),
                    reason="no host compiler or CUDA headers")
def test_larger_pyramid_at_the_old_address(tmp_path):
    flags = ["-std=c++17", "-O0", "-ffp-contract=off", "-I", CUDA_INC, "-I", CSRC]
    src, obj, main = tmp_path / "main.cpp", tmp_path / "builder.o", tmp_path / "main.o"
    src.write_text(PROGRAM)
    subprocess.run(["g++", *flags, "-c", os.path.join(CSRC, "builder.cpp"), "-o", str(obj)], check=True)
    subprocess.run(["g++", *flags, "-c", str(src), "-o", str(main)], check=True)

    def symbols(path, *args):
        out = subprocess.run(["nm", *args, str(path)], check=True, capture_output=True, text=True).stdout
        return {line.split()[-1] for line in out.splitlines() if line.strip()}

    # everything else that builder.cpp calls (launches, the runtime's other entries) does nothing
    missing = symbols(obj, "-u") - symbols(main, "--defined-only") - symbols(obj, "--defined-only")
    stubs = sorted(s for s in missing if s.startswith("_ZN2oc") or s.startswith("cuda"))
    stub = tmp_path / "stubs.c"
    stub.write_text("".join("long %s(void) { return 0; }\n" % s for s in stubs))
    subprocess.run(["gcc", "-c", str(stub), "-o", str(tmp_path / "stubs.o")], check=True)
    exe = tmp_path / "flag"
    subprocess.run(["g++", str(main), str(obj), str(tmp_path / "stubs.o"), "-ldl", "-o", str(exe)], check=True)
    assert subprocess.run([str(exe)]).returncode == 0
