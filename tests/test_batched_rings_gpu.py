"""GPU: the tcgen05 int4 projections where their rings turn over: fewer K-groups than converting sets, one more or less than stages, K slices of
unequal length, ragged columns, and every token tile's edges, against the CPU oracle's batch-1 GEMV.

Up to 32 tokens without a flag no weight is rounded: products of an fp16 activation and a small integer, at most 4608 of them summed in fp32 in
chains of at most 128 + 8 + 8 terms, so |error| <= 144 x 2^-24 x sum |x w| < 1e-5 x sqrt(K) / 4 of the row's largest value: 1e-4 covers it.  Above,
weights are rounded to fp16 (2^-11 each): the GEMV tolerance of 1e-3.
"""
import numpy as np
import pytest

import oracle.oracle as orc
from helpers import gptq_case, rel_err_max

import lithos_b200 as lb_mod

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("groups", [1, 3, 4, 5, 7, 8, 13, 36])
@pytest.mark.parametrize("N", [48, 1168])
def test_rings(ctx, lb, groups, N):
    K = 128 * groups
    qw, sc, qz, _ = gptq_case(K, N, seed=groups + N, zeros=True)
    d_w = [ctx.to_device(a) for a in (qw, sc, qz)]
    X = lb_mod.fill_normal(256 * K, groups, 41, dtype="f16").reshape(256, K)
    ref = {}
    for B in (9, 16, 17, 32, 33, 64, 65, 128, 129, 256):
        d_x, d_y = ctx.to_device(np.ascontiguousarray(X[:B])), ctx.to_device(np.full(B * N, np.nan, dtype=np.float32))
        ctx.gemm_int4(*d_w, d_x, d_y, K, N, B, lb.GEMV_Y_F32)
        y = d_y.download(np.float32, B * N).reshape(B, N)
        assert ctx.device_status() == 0 and np.isfinite(y).all()
        for b in {0, B // 2, B - 1}:
            if b not in ref:
                ref[b] = orc.gptq_gemv(qw, sc, qz, X[b], K, N)[0]
            assert rel_err_max(y[b], ref[b]) <= (1e-4 if B <= 32 else 1e-3), (B, b)
        d_x.free()
        d_y.free()
    for d in d_w:
        d.free()
