"""Compiles device code of the library for the host: the headers' functions
with CUDA's qualifiers defined away."""
import os
import shutil
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "fortress_b200", "csrc")

PRELUDE = r"""
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>
#undef __device__
#undef __host__
#undef __global__
#undef __shared__
#undef __forceinline__
#undef __align__
#define __device__
#define __host__
#define __global__
#define __shared__
#define __forceinline__ inline
#define __align__(n) alignas(n)
#define __restrict__
struct HostIndex { unsigned x, y, z; };
static HostIndex host_thread, host_block;
#define threadIdx host_thread
#define blockDim host_block
static inline unsigned __umulhi(unsigned a, unsigned b) { return (unsigned)(((unsigned long long)a * b) >> 32); }
static inline void __syncthreads() {}
static inline double rsqrt(double x) { return 1.0 / sqrt(x); }
static inline float rsqrt(float x) { return 1.0f / sqrtf(x); }
"""


CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")


def nvcc():
    path = shutil.which("nvcc") or os.path.join(CUDA, "bin", "nvcc")
    return path if os.path.exists(path) else None


def compile_probe(folder, source):
    """Path of the program made from source (its includes are of csrc).  No
    contraction: products and sums round one by one, on every host alike."""
    src, exe = folder / "probe.cpp", folder / "probe"
    src.write_text(PRELUDE + source)
    subprocess.run(["g++", "-std=c++17", "-O2", "-w", "-ffp-contract=off", "-I", os.path.join(CUDA, "include"), "-I", CSRC, "-o", str(exe),
                    str(src)], check=True, capture_output=True)
    return exe
