"""GPU: the tcgen05 int4 projections where their rings turn over: fewer K-groups than converting sets, one more or less than stages, K slices of
unequal length, with and without a K split, and every token tile's edges, against the CPU oracle's weights
(exact in fp32) times the activations in 64 bits.  Both widths end inside a warp
(N % 32 == 16: lanes without a column beside lanes with one) and inside a block of 128 columns.

Up to 32 tokens without a flag no weight is rounded: a K-group's 128 products (an fp16 activation and a small integer, exact) are summed in fp32, its scaled
sum joins at most eight others and those at most five: at most 144 roundings, each of at most 2^-23 of a partial sum (the tensor core may truncate) whose
rms is at most the row's, so the error's rms is below 144 x 2^-23 = 1.7e-5 of the row's.  Weights rounded to fp16 (2^-11 each, an rms of
2^-11 / sqrt(12) / 0.7 = 2e-4 of the row's) would not pass.  Above 32 tokens they are: the GEMV tolerance of 1e-3 of the largest value.  Results in fp16
add 2^-11 of the value.
"""
import numpy as np
import pytest

import oracle.oracle as orc
from helpers import gptq_case, rel_err_max

import lithos_b200 as lb_mod

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("groups", [1, 3, 4, 5, 7, 8, 13, 36])
@pytest.mark.parametrize("N", [48, 1168])
@pytest.mark.parametrize("zeros", [True, False])
@pytest.mark.parametrize("f32", [True, False])
def test_rings(ctx, lb, groups, N, zeros, f32):
    K = 128 * groups
    qw, sc, qz, _ = gptq_case(K, N, seed=groups + N, zeros=zeros)
    d_w = [ctx.to_device(a) if a is not None else None for a in (qw, sc, qz)]
    W = orc.gptq_dequant(qw, sc, qz, K, N).astype(np.float64)
    X = lb_mod.fill_normal(256 * K, groups, 41, dtype="f16").reshape(256, K)
    ref = {}
    for B in (9, 16, 17, 32, 33, 64, 65, 128, 129, 256):
        d_x, d_y = ctx.to_device(np.ascontiguousarray(X[:B])), ctx.to_device(np.full(B * N, np.nan, dtype=np.float32))
        ctx.gemm_int4(*d_w, d_x, d_y, K, N, B, lb.GEMV_Y_F32 if f32 else 0)
        y = d_y.download(np.float32 if f32 else np.float16, B * N).reshape(B, N)
        assert ctx.device_status() == 0 and np.isfinite(y).all()
        for b in {0, B // 2, B - 1}:
            if b not in ref:
                ref[b] = X[b].astype(np.float64) @ W
            half = 0.0 if f32 else 2.0 ** -11
            if B <= 32:
                assert np.linalg.norm(y[b] - ref[b]) / np.linalg.norm(ref[b]) <= 1.7e-5 + half, (B, b)
            assert rel_err_max(y[b], ref[b]) <= 1e-3 + half, (B, b)
        d_x.free()
        d_y.free()
    for d in d_w:
        if d:
            d.free()
