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


class View:
    def __init__(self, b, off):
        self.ptr = b.ptr + off


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


@pytest.mark.parametrize("K,N,B,tc", [
    (512, 1024, 16, False), (640, 1024, 16, True), (256, 1024, 17, False), (384, 1024, 17, True),                # short columns
    (8192, 7168, 12, False), (8192, 8832, 16, False), (8192, 9216, 9, True), (5120, 7168, 12, True),             # twice the slices, and all of them at once
    (14336, 5888, 12, False), (11008, 5888, 12, True),                                                           # four times, and idle SMs
    (1024, 9472, 16, True), (1024, 9600, 16, False), (1024, 9600, 17, True), (1024, 18944, 32, True), (1024, 18960, 32, False),
    # up to 16 tokens at widths that the ring kernels do not take, as many blocks of columns as above: what is not mma.sync here is tensor memory
    (512, 1008, 16, False), (640, 1008, 16, True), (8192, 7152, 12, False), (8192, 8816, 16, False), (8192, 9200, 9, True), (5120, 7152, 12, True),
    (14336, 5872, 12, False), (11008, 5872, 12, True), (1024, 9456, 16, True), (1024, 9584, 16, False)])
def test_which_kernel(ctx, lb, K, N, B, tc):
    """which sizes of 9 to 32 tokens have the bits of LB_GEMM_MMA_SYNC (148 SMs).  The others run on tensor memory, or, up to 16 tokens at widths in whole 32s, on the
    ring kernels; all ways are exact, so their results differ in the last bits only"""
    if ctx.sm_count != 148:
        pytest.skip("the sizes are those of 148 SMs")
    qw, sc, qz, _ = gptq_case(K, N, seed=K + N)
    d_w, d_x = [ctx.to_device(a) for a in (qw, sc, qz)], ctx.to_device(lb_mod.fill_normal(B * K, N, 42, dtype="f16"))
    got = []
    for flag in (0, lb.GEMM_MMA_SYNC):
        d_y = ctx.to_device(np.full(B * N, np.nan, dtype=np.float32))
        ctx.gemm_int4(*d_w, d_x, d_y, K, N, B, lb.GEMV_Y_F32 | flag)
        got.append(d_y.download(np.float32, B * N))
        d_y.free()
    assert ctx.device_status() == 0 and np.isfinite(got[0]).all()
    assert np.array_equal(*got) != tc
    assert np.linalg.norm(got[0] - got[1]) <= 2 * 1.7e-5 * np.linalg.norm(got[1])
    for d in (*d_w, d_x):
        d.free()


def test_rows_and_their_batch(ctx, lb):
    """what the header says of a row's bits: whoever travels with it they are the same within 2 to 8 tokens and mma.sync at 9 to 32, within 9 to 32 tokens
    on tensor memory, and from 33 tokens on; and between the first two never more than rounding apart"""
    K, N = 2048, 1168
    qw, sc, qz, _ = gptq_case(K, N, seed=5)
    d_w = [ctx.to_device(a) for a in (qw, sc, qz)]
    X = lb_mod.fill_normal(256 * K, 6, 43, dtype="f16").reshape(256, K)

    def run(rows, flag=0):
        x = np.ascontiguousarray(X[rows])
        d_x, d_y = ctx.to_device(x), ctx.to_device(np.full(len(x) * N, np.nan, dtype=np.float32))
        ctx.gemm_int4(*d_w, d_x, d_y, K, N, len(x), lb.GEMV_Y_F32 | flag)
        y = d_y.download(np.float32, len(x) * N).reshape(len(x), N)
        d_x.free()
        d_y.free()
        return y

    perm = np.random.default_rng(7).permutation(256)
    mma, tc, many = run(range(32), lb.GEMM_MMA_SYNC), run(range(32)), run(range(256))
    for B in (2, 5, 8):
        assert np.array_equal(run(range(B)), mma[:B]), B
    for B in (9, 12, 16, 17, 25):
        assert np.array_equal(run(range(B)), tc[:B]), B
        assert np.array_equal(run(range(B), lb.GEMM_MMA_SYNC), mma[:B]), B
    for B in (33, 64, 65, 128, 129, 200):
        assert np.array_equal(run(range(B)), many[:B]), B
    for B in (9, 16, 17, 32):
        assert np.array_equal(run(range(B), lb.GEMM_TCGEN05), many[:B]), B
    assert np.array_equal(run(perm[perm < 32]), tc[perm[perm < 32]]) and np.array_equal(run(perm), many[perm])
    assert np.linalg.norm(tc - mma) <= 2 * 1.7e-5 * np.linalg.norm(mma)
    assert ctx.device_status() == 0
    for d in d_w:
        d.free()


def test_alignment(ctx, lb):
    """packed words and scales on their own boundaries only (the mma.sync kernels load two at once) are taken by the exact tcgen05 kernels at any size
    up to 32 tokens, forced mma.sync refuses them, and so does every path an x beside a 16-byte boundary"""
    for K, N, sizes in ((512, 1168, (1, 2, 8, 9, 16, 17, 32, 33, 200)), (256, 48, (2, 17))):
        qw, sc, qz, _ = gptq_case(K, N, seed=N)
        W = orc.gptq_dequant(qw, sc, qz, K, N).astype(np.float64)
        X = lb_mod.fill_normal(256 * K, 8, 44, dtype="f16").reshape(256, K)
        bufs = [ctx.to_device(np.concatenate([np.zeros(1, a.dtype), a.ravel()])) for a in (qw, sc)]
        d_q, d_s = (View(b, a.itemsize) for b, a in zip(bufs, (qw, sc)))
        d_z, d_y = ctx.to_device(qz), ctx.alloc(256 * N * 4)
        for B in sizes:
            d_x = ctx.to_device(np.concatenate([np.zeros(4, np.float16), X[:B].ravel()]))
            for y32 in (lb.GEMV_Y_F32, 0):
                with pytest.raises(lb_mod.LithosError):
                    ctx.gemm_int4(d_q, d_s, d_z, View(d_x, 8), d_y, K, N, B, y32)
            if B <= 64:
                with pytest.raises(lb_mod.LithosError):
                    ctx.gemm_int4(d_q, d_s, d_z, d_x, d_y, K, N, B, lb.GEMV_Y_F32 | lb.GEMM_MMA_SYNC)
            d_x.free()
            d_x = ctx.to_device(np.ascontiguousarray(X[:B]))
            ctx.gemm_int4(d_q, d_s, d_z, d_x, d_y, K, N, B, lb.GEMV_Y_F32)
            y, want = d_y.download(np.float32, B * N).reshape(B, N), X[:B].astype(np.float64) @ W
            assert ctx.device_status() == 0
            assert np.linalg.norm(y - want) <= (1.7e-5 if B <= 32 else 1e-3) * np.linalg.norm(want), B
            d_x.free()
        for b in (*bufs, d_z, d_y):
            b.free()
