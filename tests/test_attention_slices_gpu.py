"""GPU: decode attention where its split changes: an empty cache, blocks of 16 rows and slices of 128 that are just full or just begun, few slices (merged by
one group of threads) and more than 16 (four groups), as many as make one wave and rows for several blocks per warp, every head ratio, against the CPU oracle.

Queries and probabilities enter the products as two bf16 terms (relative error 2^-17 each): a score s of up to 8 in log2 units is off by at most 8 x 2^-17, a
probability by that times ln 2 plus 2^-17, so a weighted mean of values by at most 5e-5 of the largest; the oracle's own fp32 sums over 256 features and
5000 rows add about as much.  Bound: 2e-4 of the largest value."""
import numpy as np
import pytest

from helpers import attention_case, rel_err_max

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("HQ,HKV", [(1, 1), (8, 4), (6, 2), (8, 2), (24, 4), (48, 8)])
@pytest.mark.parametrize("pos", [0, 1, 15, 16, 17, 127, 128, 129, 1024, 2049, 2320, 4735, 4737, 5003])
def test_slices(ctx, lb, oracle, HQ, HKV, pos):
    L, spare = pos + 1, 2
    c = attention_case(HQ + pos, L + spare, HQ, HKV)
    f = oracle.bf16_to_f32
    kc, vc = c["kc"].copy(), c["vc"].copy()
    want = oracle.attention_step(f(c["q"]), f(c["k_new"]), f(c["v_new"]), f(c["gate"]), f(c["q_norm_w"]), f(c["k_norm_w"]), kc, vc, pos, HQ, HKV)
    d = {n: ctx.to_device(c[n]) for n in c}
    got = []
    for _ in range(2):
        o = ctx.to_device(np.full(HQ * 256, np.nan, np.float32))
        ctx.attention_decode(d["q"], d["k_new"], d["v_new"], d["gate"], d["q_norm_w"], d["k_norm_w"], d["kc"], d["vc"], o, pos, HQ, HKV)
        got.append(o.download(np.float32, HQ * 256))
        o.free()
    assert ctx.device_status() == 0
    assert np.array_equal(*got)
    assert rel_err_max(got[0], want.ravel()) <= 2e-4
    k, v = (d[n].download(np.uint16, (L + spare) * HKV * 256).reshape(L + spare, HKV, 256) for n in ("kc", "vc"))
    assert np.array_equal(v, vc) and np.array_equal(np.delete(k, pos, 0), np.delete(kc, pos, 0))  # the new row and nothing else
    for x in d.values():
        x.free()


@pytest.mark.parametrize("HQ,HKV,pos", [(24, 4, 300), (24, 4, 4096), (8, 4, 2049), (48, 8, 5003), (6, 1, 9000), (4, 2, 9472)])
def test_shares_left_to_the_last_arrival(ctx, lb, HQ, HKV, pos):
    """No CTA waits for others that may not be resident: one that has waited for its limit leaves its share to the last to arrive, the result is the same and
    nothing is reported.  With a limit of a nanosecond nearly every CTA leaves, with the built-in one hardly any does; calls alternate, since the words reset themselves."""
    c = attention_case(HQ + pos, pos + 2, HQ, HKV)
    d = {n: ctx.to_device(c[n]) for n in c}
    got = []
    for limit in (0, 1, 1, 0, 1):
        ctx.set_wait_limit(limit)
        for _ in range(4):
            o = ctx.to_device(np.full(HQ * 256, np.nan, np.float32))
            ctx.attention_decode(d["q"], d["k_new"], d["v_new"], d["gate"], d["q_norm_w"], d["k_norm_w"], d["kc"], d["vc"], o, pos, HQ, HKV)
            got.append(o.download(np.float32, HQ * 256))
            o.free()
    ctx.set_wait_limit(0)
    assert ctx.device_status() == 0 and np.isfinite(got[0]).all()
    for g in got[1:]:
        assert np.array_equal(g, got[0])
    for x in d.values():
        x.free()


@pytest.mark.parametrize("HQ,HKV", [(4, 1), (6, 2)])
@pytest.mark.parametrize("pos", [8193, 9473, 20000])
@pytest.mark.parametrize("late", [False, True])
def test_more_slices_than_one_trip(ctx, lb, oracle, HQ, HKV, pos, late):
    """one or two KV heads have more than 64 slices, which are added in two trips or three: a head's largest score in the first slice or in the last one, about as
    heavy as all other rows together, so that what was summed before, or what comes after, is brought to another maximum (features that do not rotate).  The bound
    above, with a largest score of 16 in place of 8: 4e-4."""
    c = attention_case(HQ + pos, pos + 3, HQ, HKV)
    f = oracle.bf16_to_f32
    q, kc = f(c["q"]).reshape(HQ, 256), c["kc"]
    row = pos - 3 if late else 5
    for kv in range(HKV):
        k = np.zeros(256, np.float32)
        h = q[kv * (HQ // HKV)]
        k[64:] = h[64:] * (10.0 * 16.0 / np.sum(h[64:] ** 2))
        kc[row, kv] = lb.f32_to_bf16(k)
    kw, vw = kc.copy(), c["vc"].copy()
    want = oracle.attention_step(f(c["q"]), f(c["k_new"]), f(c["v_new"]), f(c["gate"]), f(c["q_norm_w"]), f(c["k_norm_w"]), kw, vw, pos, HQ, HKV)
    d = {n: ctx.to_device(c[n]) for n in c}
    o = ctx.to_device(np.full(HQ * 256, np.nan, np.float32))
    ctx.attention_decode(d["q"], d["k_new"], d["v_new"], d["gate"], d["q_norm_w"], d["k_norm_w"], d["kc"], d["vc"], o, pos, HQ, HKV)
    got = o.download(np.float32, HQ * 256)
    assert ctx.device_status() == 0
    assert rel_err_max(got, want.ravel()) <= 4e-4
    for x in (*d.values(), o):
        x.free()
