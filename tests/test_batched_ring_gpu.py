"""GPU: int4 projections of 2 to 16 tokens on the ring kernels: fewer K-groups than warps, as many as slots and one more, K slices of unequal length, column
blocks of 32, 96 and 128, more of them than SMs, with and without zero-points, both result types, a result beside a 16-byte boundary; a row's bits do not depend on how many
travel with it (2 to 16), nor on the run.

No weight is rounded: a K-group's 128 products (an fp16 activation and a small integer, exact) are summed in fp32, its scaled sum joins at most 16 others of its
warp, then at most 8 warps' and 8 slices': at most 160 roundings of at most 2^-23 of a partial sum (the tensor core may truncate) whose rms is at most the row's,
so below 160 x 2^-23 = 1.9e-5 of the row's rms.  Results in fp16 add 2^-11."""
import numpy as np
import pytest

import oracle.oracle as orc
from helpers import gptq_case

import lithos_b200 as lb_mod

pytestmark = pytest.mark.gpu


class View:
    def __init__(self, b, off):
        self.ptr = b.ptr + off


@pytest.mark.parametrize("groups,N", [(g, n) for g in (1, 3, 8, 9, 16, 17, 18, 21, 22, 45) for n in (32, 1184)] + [(5, 96), (45, 96), (9, 9600), (2, 18976)])
@pytest.mark.parametrize("zeros", [True, False])
def test_ring(ctx, lb, groups, N, zeros):
    K = 128 * groups
    qw, sc, qz, _ = gptq_case(K, N, seed=groups + N, zeros=zeros)
    d_w = [ctx.to_device(a) if a is not None else None for a in (qw, sc, qz)]
    W = orc.gptq_dequant(qw, sc, qz, K, N).astype(np.float64)
    X = lb_mod.fill_normal(16 * K, groups, 46, dtype="f16").reshape(16, K)
    ref = X.astype(np.float64) @ W

    def run(rows, flag, off=0):
        E = 4 if flag else 2
        d_x, d_y = ctx.to_device(np.ascontiguousarray(X[rows])), ctx.to_device(np.full(len(rows) * N + 4, np.nan, dtype=np.float32))
        ctx.gemm_int4(*d_w, d_x, View(d_y, off), K, N, len(rows), flag)
        y = d_y.download(np.float32 if flag else np.float16, len(rows) * N, off).reshape(len(rows), N)
        assert ctx.device_status() == 0 and E * y.size == y.nbytes
        d_x.free()
        d_y.free()
        return y

    few = run(range(8), lb.GEMV_Y_F32)
    for B in (2, 5, 8, 9, 12, 16):
        y = run(range(B), lb.GEMV_Y_F32)
        assert np.linalg.norm(y - ref[:B]) <= 1.9e-5 * np.linalg.norm(ref[:B]), B
        assert np.array_equal(y, run(range(B), lb.GEMV_Y_F32, 4))
        if B <= 8:
            assert np.array_equal(y, few[:B]), B
        h = run(range(B), 0)
        assert np.array_equal(h, y.astype(np.float16)), B
    perm = [7, 3, 0, 5]
    assert np.array_equal(run(perm, lb.GEMV_Y_F32), few[perm])
    if groups > 8 and N <= 1184:  # sizes at which 9 to 16 tokens run on it too
        y = run(range(16), lb.GEMV_Y_F32)
        assert np.array_equal(y[:8], few)
    for d in d_w:
        if d:
            d.free()
