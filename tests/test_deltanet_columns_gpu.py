"""GPU: runs of DeltaNet steps in the kernels of 32 and of 16 columns per CTA (head counts on either side of the rule, more than eight steps, whole and
broken runs of eight): the bits of the same steps in runs of at most eight, and the oracle's values to fp32 rounding (sums of 128 terms: 1e-5)."""
import numpy as np
import pytest

from helpers import deltanet_case, rel_err_max

pytestmark = pytest.mark.gpu


class View:
    def __init__(self, b, off=0):
        self.ptr = b.ptr + off


@pytest.mark.parametrize("HV,HK", [(16, 8), (24, 8), (32, 16), (48, 16), (64, 16), (96, 32)])
@pytest.mark.parametrize("T", [9, 13, 16, 21, 40])
@pytest.mark.parametrize("f32", [False, True])
def test_runs(ctx, lb, oracle, HV, HK, T, f32):
    c = deltanet_case(3 + T, HV, HK, steps=T)
    g, beta = np.empty((T, HV), np.float32), np.empty((T, HV), np.float32)
    for t in range(T):
        g[t], beta[t] = oracle.decay_gate(c["a"][t], c["a_log"], c["dt_bias"], c["b"][t])
    f = [oracle.bf16_to_f32(c[n]) for n in ("q", "k", "v")]
    state, want = c["state"].copy(), np.empty((T, HV, 128), np.float32)
    q, k, v = (x.reshape(T, -1, 128) for x in f)
    for t in range(T):
        want[t] = oracle.deltanet_step(state, q[t], k[t], v[t], None, g[t], beta[t], HV, HK)
    E, d = (4, [ctx.to_device(x) for x in f]) if f32 else (2, [ctx.to_device(c[n]) for n in ("q", "k", "v")])
    d_g, d_b, got = ctx.to_device(g), ctx.to_device(beta), []
    for step in (T, 8):
        s, o = ctx.to_device(c["state"]), ctx.alloc(want.nbytes)
        for t in range(0, T, step):
            ctx.deltanet_step(s, View(d[0], t * HK * 128 * E), View(d[1], t * HK * 128 * E), View(d[2], t * HV * 128 * E), None, View(d_g, t * HV * 4), View(d_b, t * HV * 4),
                              View(o, t * HV * 512), HV, HK, n_steps=min(step, T - t), in_is_f32=f32)
        got.append((o.download(np.float32, want.size), s.download(np.float32, state.size)))
    assert np.array_equal(got[0][0], got[1][0]) and np.array_equal(got[0][1], got[1][1])
    assert rel_err_max(got[0][0], want.ravel()) <= 1e-5 and rel_err_max(got[0][1], state.ravel()) <= 1e-5
