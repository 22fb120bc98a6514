"""GPU: the two launch shapes of the int4 GEMV (two CTAs an SM with a deep ring, or shared memory for four): slices longer than the ring, exactly as long and shorter,
cluster counts that fit and one too many, a ragged last slice and column tile; and chains of launches in which each reads what the one before wrote while the next is let in
early.  Against the dequantised weights in 64 bits: sums of at most 136 groups in fp32, 136 x 2^-24 = 8e-6 of the row's rms."""
import numpy as np
import pytest

import oracle.oracle as orc
from helpers import gptq_case

import lithos_b200 as lb_mod

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("K,N", [(5120, 16384), (5120, 10240), (3072, 11008), (1664, 14592), (17408, 1056), (2560, 34816)])
def test_plans(ctx, lb, K, N):
    qw, sc, qz, _ = gptq_case(K, N, seed=K + N, zeros=True)
    d_w = [ctx.to_device(a) for a in (qw, sc, qz)]
    x = lb_mod.fill_normal(K, 3, 5, dtype="f16")
    d_x, d_y = ctx.to_device(x), ctx.to_device(np.full(N, np.nan, dtype=np.float32))
    for _ in range(3):  # behind itself
        ctx.gemv_int4(*d_w, d_x, d_y, K, N, lb.GEMV_Y_F32)
    y = d_y.download(np.float32, N)
    assert ctx.device_status() == 0
    W = orc.gptq_dequant(qw, sc, qz, K, N)
    ref = np.concatenate([x.astype(np.float64) @ W[:, i:i + 2048].astype(np.float64) for i in range(0, N, 2048)])
    assert np.linalg.norm(y - ref) <= 1e-5 * np.linalg.norm(ref)


def test_chain_of_launches(ctx, lb):
    K = 8192
    qw, sc, qz, _ = gptq_case(K, K, seed=8, zeros=True)
    d_w = [ctx.to_device(a) for a in (qw, sc, qz)]
    x = (lb_mod.fill_normal(K, 4, 5, dtype="f32") * 1e-3).astype(np.float16)

    def run(wait):
        b = [ctx.to_device(x), ctx.to_device(np.zeros(K, dtype=np.float16))]
        for i in range(8):
            ctx.gemv_int4(*d_w, b[i & 1], b[1 - (i & 1)], K, K, 0)
            if wait:
                ctx.sync()
        return b[0].download(np.float16, K)

    want = run(True)
    assert np.isfinite(want).all() and np.abs(want).max() > 0
    for _ in range(5):
        assert np.array_equal(run(False).view(np.uint16), want.view(np.uint16))
    assert ctx.device_status() == 0
