"""GPU: a run of DeltaNet steps is its steps one by one, bit for bit, whatever its length (one step and two have kernels of their own; runs of
eight tokens, read-outs four at a time), and both are the oracle's to fp32 rounding (sums of 128 terms, 2^-24 each, errors shrink with the state: 1e-5 of the largest value)."""
import numpy as np
import pytest

from helpers import deltanet_case, rel_err_max

pytestmark = pytest.mark.gpu


class View:
    def __init__(self, b, off=0):
        self.ptr = b.ptr + off


@pytest.mark.parametrize("T", [1, 2, 3, 4, 5, 7, 8, 9, 16, 23])
@pytest.mark.parametrize("heads", [(3, 1), (4, 2), (2, 2), (76, 4)])  # 76: more CTAs than two per SM, so two steps take the run's kernel
@pytest.mark.parametrize("f32", [False, True])
@pytest.mark.parametrize("off", [0, 4])  # the state on an 8-byte boundary and beside one
def test_run_equals_steps(ctx, lb, oracle, T, heads, f32, off):
    HV, HK = heads
    c = deltanet_case(5 + T, HV, HK, steps=T)
    g, beta = np.empty((T, HV), np.float32), np.empty((T, HV), np.float32)
    for t in range(T):
        g[t], beta[t] = oracle.decay_gate(c["a"][t], c["a_log"], c["dt_bias"], c["b"][t])
    qf, kf, vf = (oracle.bf16_to_f32(c[n]).reshape(T, -1, 128) for n in ("q", "k", "v"))
    z = lb.fill_normal(T * HV * 128, 9, 9).reshape(T, HV, 128) if T % 2 else None
    state, want = c["state"].copy(), np.empty((T, HV, 128), np.float32)
    for t in range(T):
        want[t] = oracle.deltanet_step(state, qf[t], kf[t], vf[t], z[t] if z is not None else None, g[t], beta[t], HV, HK)
    E, d = (4, [ctx.to_device(a) for a in (qf, kf, vf)]) if f32 else (2, [ctx.to_device(c[n]) for n in ("q", "k", "v")])
    d_g, d_b, d_z = ctx.to_device(g), ctx.to_device(beta), ctx.to_device(z) if z is not None else None
    got = []
    for one in (False, True):
        s, o = ctx.to_device(np.concatenate([np.zeros(off // 4, np.float32), c["state"].ravel()])), ctx.alloc(want.nbytes)
        if one:
            for t in range(T):
                ctx.deltanet_step(View(s, off), View(d[0], t * HK * 128 * E), View(d[1], t * HK * 128 * E), View(d[2], t * HV * 128 * E),
                                  View(d_z, t * HV * 512) if d_z else None, View(d_g, t * HV * 4), View(d_b, t * HV * 4), View(o, t * HV * 512), HV, HK, in_is_f32=f32)
        else:
            ctx.deltanet_step(View(s, off), *d, d_z, d_g, d_b, o, HV, HK, n_steps=T, in_is_f32=f32)
        got.append((o.download(np.float32, want.size), s.download(np.float32, state.size, off)))
    assert np.array_equal(got[0][0], got[1][0]) and np.array_equal(got[0][1], got[1][1])
    assert rel_err_max(got[0][0], want.ravel()) <= 1e-5 and rel_err_max(got[0][1], state.ravel()) <= 1e-5
