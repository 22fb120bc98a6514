"""GPU: the bounded mbarrier waits of the tensor-core kernels.  A wait for a barrier that nobody arrives at gives up after LB_WAIT_NS (2 s) or its number of
polls, whichever is first, and says so: a poll may suspend the thread for as long as the hardware likes, so polls alone are no bound.  A wait for a
completed barrier succeeds at once.  3 s allow for the polls between two readings of the clock."""
import ctypes as C
import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
KERNELS = Path(__file__).resolve().parent.parent / "lithos_b200" / "csrc" / "kernels"
SOURCE = """
#include "tcgen05.cuh"
extern "C" __global__ void waits(unsigned long long* out) { // [warp]: nanoseconds, [8 + warp]: result; warps 0-2: no arrival, 3-5: one before the wait
    __shared__ __align__(8) uint64_t bar[6];
    const int warp = threadIdx.x >> 5;
    if (threadIdx.x == 0) {
        for (int i = 0; i < 6; ++i) mbar_init(&bar[i], 1);
        mbar_fence_init();
        for (int i = 3; i < 6; ++i) mbar_arrive(&bar[i]);
    }
    __syncthreads();
    if ((threadIdx.x & 31) == 0) {
        const uint64_t t = globaltimer_ns();
        const bool ok = warp % 3 == 0 ? mbar_wait(&bar[warp], 0) : warp % 3 == 1 ? tc_wait(&bar[warp], 0) : tc2_wait(&bar[warp], 0);
        out[warp] = globaltimer_ns() - t;
        out[8 + warp] = ok;
    }
}
"""


def test_waits_end(ctx, lb, tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    src, cubin = tmp_path / "waits.cu", tmp_path / "waits.cubin"
    src.write_text(SOURCE)
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-I", str(KERNELS), "-cubin", "-o", str(cubin), str(src)], check=True)
    L = lb.lib()
    L.lb_module_load.argtypes = [C.c_void_p, C.c_char_p, C.POINTER(C.c_int)]
    L.lb_module_get_kernel.argtypes = [C.c_void_p, C.c_int, C.c_char_p, C.POINTER(C.c_uint64)]
    L.lb_launch_kernel.argtypes = [C.c_void_p, C.c_uint64] + [C.c_uint] * 7 + [C.POINTER(C.c_void_p)]
    mod, fn = C.c_int(), C.c_uint64()
    ctx._check(L.lb_module_load(ctx.h, str(cubin).encode(), C.byref(mod)))
    ctx._check(L.lb_module_get_kernel(ctx.h, mod, b"waits", C.byref(fn)))
    out = ctx.alloc(16 * 8)
    p = C.c_uint64(out.ptr)
    ctx._check(L.lb_launch_kernel(ctx.h, fn, 1, 1, 1, 192, 1, 1, 0, (C.c_void_p * 1)(C.addressof(p))))
    ctx.sync()
    r = out.download(np.uint64, 16)
    out.free()
    assert list(r[8:14]) == [0, 0, 0, 1, 1, 1]
    assert (r[:3] <= 3_000_000_000).all() and (r[3:6] <= 1_000_000).all(), r
