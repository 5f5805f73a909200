"""A pass that cannot be launched ends its call with an error.

The launchers of the size-specialised passes refuse lengths without a kernel
by their return value alone, and a failed grouped pass is known only from its
launcher.  The library's host code is compiled with a program that asks for
such passes (no GPU is used) and has to get the refusal back from launch_row,
launch_col and group_step.  Where the unfused FFT and BFT may take the
size-specialised column passes, they have to ask for them as well."""
import os
import subprocess

import pytest

from tests.host_device import CSRC, nvcc

PROBE = r"""
#include "fgpe_api.cu"
#include <cstdio>
template <typename T, int MS> int refused() {
    fgpe_s h;
    memset(&h.p, 0, sizeof h.p);
    h.p.dim = 3; h.p.nx = h.p.ny = h.p.nz = 100;          // no size-specialised kernel
    h.ms = MS; h.fp32 = sizeof(T) == 4; h.npts = 1000000;
    int bad = 0;
    h.fast_row = h.fast_col[1] = h.fast_col[2] = true;
    cudaGetLastError();
    if (launch_row<T, MS>(&h, ROW_FULL, nullptr) == cudaSuccess) bad |= 1;
    h.warp_row = true;
    if (launch_row<T, MS>(&h, ROW_FULL, nullptr) == cudaSuccess) bad |= 2;
    h.warp_row = false;
    h.reg_row = true;
    if (launch_row<T, MS>(&h, ROW_FULL, nullptr) == cudaSuccess) bad |= 4;
    if (launch_col<T, MS>(&h, 1, COL_SCALE | COL_FWD | COL_STEP) == cudaSuccess) bad |= 8;
    if (launch_col<T, MS>(&h, 2, COL_FWD | COL_KOP | COL_INV | COL_STEP) == cudaSuccess) bad |= 16;
    // single transforms outside a step go to the same launchers, not to the
    // pass of any length
    h.plain[1] = h.plain[2] = true;
    if (launch_col<T, MS>(&h, 1, COL_FWD) != cudaErrorInvalidValue) bad |= 128;
    if (launch_col<T, MS>(&h, 2, COL_INV) != cudaErrorInvalidValue) bad |= 256;
    BatchGroup g;
    g.nx = 128; g.ny = 100; g.ms = MS; g.fp32 = h.fp32;
    g.members.push_back(0);
    if (group_step(g, 0, nullptr) == cudaSuccess) bad |= 32;
    g.nx = 100; g.ny = 128;
    if (group_step(g, 0, nullptr) == cudaSuccess) bad |= 64;
    return bad;
}
int main() {
    std::printf("%d %d %d %d\n", refused<float, 3>(), refused<float, 5>(), refused<double, 3>(), refused<double, 5>());
    return 0;
}
"""


def test_refused_passes_are_reported(tmp_path):
    lib = os.path.dirname(CSRC)
    if not nvcc() or not os.path.exists(os.path.join(lib, "libfgpe.so")):
        pytest.skip("needs nvcc and the built library")
    (tmp_path / "probe.cu").write_text(PROBE)
    exe = tmp_path / "probe"
    # -G: device code is not run, and compiles fastest without optimisation
    subprocess.run([nvcc(), "-std=c++17", "-G", "--expt-relaxed-constexpr", "-gencode", "arch=compute_100a,code=sm_100a", "-w",
                    "-I", CSRC, "-o", str(exe), str(tmp_path / "probe.cu"), "-L", lib, "-lfgpe", "-Xlinker", "-rpath," + lib],
                   check=True, capture_output=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout
    assert out.split() == ["0"] * 4, out
