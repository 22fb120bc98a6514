"""GPU: prompts through the state-space recurrence on the 5th-generation tensor cores (states of up to 128 rows and heads of 33 to 64 columns after padding): blocks
of 128 tokens, ragged last ones, one segment and several, groups of heads, columns that are not whole 16-byte pieces, decays from fast to nearly none.  Logits
against oracle/vobunex.py with the bounds of the models' own tests; the states of a whole prompt and of portions (short ones take the other kernel) within 1e-2 of
their largest value (the convolution's outputs are bf16: 2^-9 each)."""
import numpy as np
import pytest

import test_vobunex_gpu as TV
import vobunex_cases as CV

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("heads,vdim,state,groups", [(2, 64, 128, 1), (6, 60, 120, 2), (4, 33, 113, 4), (3, 48, 128, 3), (80, 64, 128, 8)])
def test_chunk(ctx, lb, tmp_path, heads, vdim, state, groups):
    c = TV.Case(tmp_path, ctx, CV.config(64, 61, [CV.mamba2(heads, vdim, state, groups=groups), CV.mamba2(heads, vdim, state, groups=groups, mlp=CV.dense(40))]), heads + vdim)
    n = 900 if heads < 80 else 520
    toks = TV.tokens(c.cfg, n, 6)
    want = c.want(toks)
    m = c.open("bfloat16", n)
    states = []
    for cuts in ([n], [65, 1, 127, 129, n - 322], [128, 256, 64, n - 448], [255, 30, n - 285]):
        m.reset_state()
        TV.check(TV.feed(m, toks, cuts), want, "bfloat16", cuts)
        states.append(m.get_state(0, 0, np.float32, heads * state * vdim))
    for s in states[1:]:
        assert np.isfinite(s).all() and np.max(np.abs(s - states[0])) <= 1e-2 * np.max(np.abs(states[0]))
    assert ctx.device_status() == 0
    m.close()


def test_little_forgetting(ctx, lb, tmp_path):
    """heads that hardly forget, and heads that forget within a token: sums of log decays over a block from nearly 0 to some hundreds"""
    def tweak(w):
        for k in w:
            if k.endswith("a_log") or "A_log" in k:
                w[k] = np.resize(np.array([-7.0, 3.0], np.float32), w[k].shape)
    c = TV.Case(tmp_path, ctx, CV.config(64, 61, [CV.mamba2(4, 64, 128, groups=2), CV.mamba2(4, 64, 128)]), 9, tweak)
    toks = TV.tokens(c.cfg, 700, 3)
    want = c.want(toks)
    m = c.open("bfloat16", 700)
    for cuts in ([700], [300, 400]):
        m.reset_state()
        TV.check(TV.feed(m, toks, cuts), want, "bfloat16", cuts)
    assert ctx.device_status() == 0
    m.close()
