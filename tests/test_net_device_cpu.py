"""A net does its work on the device that was current when it was made, whichever is current later, and its run's status is that of
the step that failed: the library against a CUDA runtime that only keeps book of devices and launches (no GPU)."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

RUNTIME = r"""
#include <stdio.h>
#include <string.h>
static int current = 0, launches[2], opened[2];
extern "C" {
int cudaGetDevice(int* d) { *d = current; return 0; }
int cudaSetDevice(int d) { current = d; return 0; }
int cudaDeviceGetAttribute(int* v, int attr, int) { *v = attr == 16 ? 148 : 232448; return 0; }      // cudaDevAttrMultiProcessorCount
int cudaGetSymbolAddress(void** p, const void*) { static int word; *p = &word; return 0; }
int cudaFuncSetAttribute(const void*, int, int) { ++opened[current]; return 0; }
int cudaLaunchKernelExC(const void*, const void*, void**) { ++launches[current]; return 0; }
}
"""

PROGRAM = r"""
#include <stdlib.h>
#include "tdc_b200.h"
#define MUST(e) do { if ((e) != 0) { printf("%s: %s\n", #e, tdc_last_error_string()); return 1; } } while (0)
int main() {
    static float w[64 * 16 * 9], fc[10 * 64], x[16 * 64], y[64 * 64];
    tdc_net* n;
    cudaSetDevice(1);
    MUST(tdc_net_create(&n, 20, 16, 8, 8));
    int t;
    MUST(tdc_net_pack(n, TDC_NET_PACK, &t));
    tdc_net_conv d{};
    d.kind = TDC_NET_CONV3x3; d.K = 64; d.residual = d.into = -1; d.out = TDC_NET_PLANES;
    MUST(tdc_net_conv_plan(n, t, &d));
    d.filter = w;
    cudaSetDevice(0);
    MUST(tdc_net_add_conv(n, t, &d, &t));
    MUST(tdc_net_head(n, t, nullptr, nullptr, fc, nullptr, 10));
    size_t bytes;
    MUST(tdc_net_finish(n, &bytes));
    void* arena = aligned_alloc(256, (bytes + 255) / 256 * 256);
    MUST(tdc_net_run(n, x, nullptr, y, nullptr, arena, bytes, nullptr));
    printf("opened %d %d launches %d %d current %d\n", opened[0], opened[1], launches[0], launches[1], current);
    tdc_net_destroy(n);
    // a step that its entry point refuses: the run's status is that refusal
    MUST(tdc_net_create(&n, 1, 16, 8, 8));
    tdc_net_nchw c{};
    c.K = 8; c.R = c.S = 1; c.stride = 3; c.filter = w; c.residual = -1; c.to_y = 1;
    MUST(tdc_net_nchw_conv(n, -1, &c, &t));
    MUST(tdc_net_finish(n, &bytes));
    const int rc = tdc_net_run(n, x, nullptr, y, nullptr, x, bytes, nullptr);
    printf("status %d %s\n", rc, tdc_last_error_string());
    return 0;
}
"""


def test_the_device_of_a_net(built, tmp_path):
    objs = [os.path.join(ROOT, "ppopp23-tdc_b200", "build", f + ".o") for f in ("net", "conv_pk", "abi", "conv_tc", "conv_f32_gemm", "tile", "pool", "affine", "inst_1x1", "inst_3x3s1", "inst_3x3s2", "inst_rt", "layers")]
    if not all(os.path.exists(o) for o in objs):
        pytest.skip("the library's object files are not here")
    src = tmp_path / "device.cpp"
    src.write_text(RUNTIME + PROGRAM)
    exe = str(tmp_path / "device")
    r = subprocess.run(["nvcc", "-std=c++17", "-cudart", "shared", "-I", os.path.join(ROOT, "include"), "-o", exe, str(src), *objs, "-Xlinker", "--allow-multiple-definition"], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([exe], capture_output=True, text=True)
    lines = r.stdout.split("\n")
    assert r.returncode == 0 and lines[0] == "opened 0 2 launches 0 4 current 0", r.stdout + r.stderr
    assert lines[1].startswith("status 3 stride 3"), r.stdout


def test_images_whose_positions_do_not_count_in_32_bits_are_refused(built):
    """50000 x 50000 positions overflow an int, and the sizes computed from it would pass every later check."""
    import ctypes as C
    from tdc_b200 import _lib
    h, d = C.c_void_p(), _lib.NetConv()
    for B, H, W in ((1, 50000, 50000), (1, 1 << 30, 4), (4096, 1024, 1024)):
        assert _lib.lib.tdc_net_create(C.byref(h), B, 1, H, W) == _lib.ERR_SHAPE and not h
        assert _lib.lib.tdc_net_estimate(B, 16, H, W, 0, C.byref(d)) == _lib.ERR_SHAPE
