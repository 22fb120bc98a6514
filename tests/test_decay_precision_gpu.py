"""GPU: decays and betas of a prompt (pf_ab_gate, both block shapes) against 64 bits, from the kernels' own outputs: a loss of precision there would drown in the
logits' tolerance.  The operands (fp16 activations, bf16 rows) are exact in the products, so what remains is the order and rounding of the fp32 sums and the
exponentials: the rms distance is at most three times that of the same formulas with numpy's fp32 sums and fp32 exponentials, whose bound per operation is the same
2^-24 (the tensor core may truncate: 2^-23, hence two, and one more for the device's exponentials of 2 ulp).  One chain of products over all of the hidden size is ten times as far off."""
import ctypes as C
from pathlib import Path

import numpy as np
import pytest

import lithos_b200 as lb_mod

pytestmark = pytest.mark.gpu
CUBIN = Path(__file__).resolve().parent.parent / "lithos_b200" / "kernels" / "prefill.cubin"


@pytest.mark.parametrize("HV,H,T", [(48, 5120, 75), (48, 5120, 200), (6, 1024, 7), (20, 1152, 33)])
@pytest.mark.parametrize("entry,rows", [("pf_ab_gate", 24), ("pf_ab_gate_few", 8)])
def test_against_64_bits(ctx, lb, entry, rows, HV, H, T):
    L = lb.lib()
    L.lb_module_load.argtypes = [C.c_void_p, C.c_char_p, C.POINTER(C.c_int)]
    L.lb_module_get_kernel.argtypes = [C.c_void_p, C.c_int, C.c_char_p, C.POINTER(C.c_uint64)]
    L.lb_launch_kernel.argtypes = [C.c_void_p, C.c_uint64] + [C.c_uint] * 7 + [C.POINTER(C.c_void_p)]
    mod, fn = C.c_int(), C.c_uint64()
    ctx._check(L.lb_module_load(ctx.h, str(CUBIN).encode(), C.byref(mod)))
    ctx._check(L.lb_module_get_kernel(ctx.h, mod, entry.encode(), C.byref(fn)))
    x = lb_mod.fill_normal(T * H, 1, 1, dtype="f16").reshape(T, H)
    w = [lb_mod.fill_normal(HV * H, 1, 2 + i, std=0.02, dtype="bf16").reshape(HV, H) for i in range(2)]
    a_log, dt = lb_mod.fill_uniform(HV, 1, 4, 0.0, 2.7), lb_mod.fill_normal(HV, 1, 5, std=0.1, dtype="bf16")
    chan = 128
    proj = lb_mod.fill_normal(T * chan, 1, 6).reshape(T, chan)
    d = [ctx.to_device(v) for v in (x, *w, a_log, dt)]
    d_g, d_b = (ctx.to_device(np.full(T * HV, np.nan, np.float32)) for _ in range(2))
    d_p, d_r = ctx.to_device(proj), ctx.to_device(np.zeros(4 * chan, np.float32))
    vals = [C.c_uint64(b.ptr) for b in (*d, d_g, d_b)] + [C.c_int(HV), C.c_int(H), C.c_int(T), C.c_uint64(d_p.ptr), C.c_int(chan), C.c_uint64(d_r.ptr), C.c_int(chan), C.c_int(3)]
    params = (C.c_void_p * len(vals))(*[C.cast(C.pointer(v), C.c_void_p) for v in vals])
    ctx._check(L.lb_launch_kernel(ctx.h, fn, (T + 15) // 16, (2 * HV + rows - 1) // rows, 1, 256, 1, 1, 0, params))
    g, beta = (b.download(np.float32, T * HV).reshape(T, HV) for b in (d_g, d_b))
    assert ctx.device_status() == 0
    a, b = (x.astype(np.float64) @ lb_mod.bf16_to_f32(m).reshape(HV, H).astype(np.float64).T for m in w)
    want_g = np.exp(-np.exp(a_log.astype(np.float64)) * np.logaddexp(0.0, a + lb_mod.bf16_to_f32(dt).astype(np.float64)))
    want_b = 1.0 / (1.0 + np.exp(-b))
    a32, b32 = (x.astype(np.float32) @ lb_mod.bf16_to_f32(m).reshape(HV, H).T for m in w)
    g32 = np.exp(-np.exp(a_log) * np.log1p(np.exp(a32 + lb_mod.bf16_to_f32(dt))))
    rms = lambda p, q: float(np.sqrt(np.mean((p.astype(np.float64) - q) ** 2)))  # noqa: E731
    own, fp32 = (rms(g, want_g), rms(beta, want_b)), (rms(g32, want_g), rms(np.float32(1) / (np.float32(1) + np.exp(-b32)), want_b))
    assert own[0] <= 3 * fp32[0] and own[1] <= 3 * fp32[1], (own, fp32)
    ring = d_r.download(np.float32, 4 * chan).reshape(4, chan)
    for s in range(max(0, T - 4), T):
        assert np.array_equal(ring[(3 + s) & 3], proj[s])
    for v in (*d, d_g, d_b, d_p, d_r):
        v.free()
