"""GPU: the int4 projections of 33 to 256 tokens carry as many tokens as there are, in steps of 16: around every step where the stages change (64, 128, 160
tokens) and beside it, a row has the bits it has among 256 tokens, and those are the oracle's weights, rounded to fp16, times the activations
(2^-11 per weight, rms 2^-11 / sqrt(12) / 0.7 = 2e-4 of a row's rms; five times that for the largest of 1168 values)."""
import numpy as np
import pytest

import oracle.oracle as orc
from helpers import gptq_case

import lithos_b200 as lb_mod

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("K,N", [(128, 48), (1152, 1168), (2048, 256)])
def test_token_steps(ctx, lb, K, N):
    qw, sc, qz, _ = gptq_case(K, N, seed=K + N)
    d_w = [ctx.to_device(a) for a in (qw, sc, qz)]
    W = orc.gptq_dequant(qw, sc, qz, K, N).astype(np.float64)
    X = lb_mod.fill_normal(256 * K, K, 45, dtype="f16").reshape(256, K)
    many = None
    for B in (256, 33, 47, 48, 49, 64, 65, 80, 81, 97, 112, 128, 129, 144, 145, 160, 161, 176, 177, 192, 208, 224, 241):
        d_x, d_y = ctx.to_device(np.ascontiguousarray(X[:B])), ctx.to_device(np.full(B * N, np.nan, dtype=np.float32))
        ctx.gemm_int4(*d_w, d_x, d_y, K, N, B, lb.GEMV_Y_F32)
        y = d_y.download(np.float32, B * N).reshape(B, N)
        assert ctx.device_status() == 0
        if many is None:
            many, want = y, X.astype(np.float64) @ W
            assert np.max(np.abs(y - want)) <= 1e-3 * np.max(np.abs(want))
        assert np.array_equal(y, many[:B]), B
        d_x.free()
        d_y.free()
    for d in d_w:
        d.free()
