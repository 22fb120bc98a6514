"""GPU: prompts through the recurrences with a decay per channel, in segments that run side by side: one to eight segments, last ones of a few tokens, every kernel
(64, 128, 256 rows), value widths that are not whole 16-byte pieces or whole slabs.  Logits against oracle/nufalorn.py with the bounds of the models' own tests;
the states of a whole prompt and of portions (other segments) within 2e-5 of their largest value (fp32 sums over at most 400 tokens, as test_nufalorn_gpu.py)."""
import numpy as np
import pytest

import nufalorn_cases as C
import test_nufalorn_gpu as TN

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("heads,dk,dv", [(3, 64, 64), (2, 50, 70), (4, 128, 128), (3, 100, 116), (2, 128, 33), (2, 256, 100), (1, 160, 64)])
@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_segments(ctx, lb, tmp_path, heads, dk, dv, dtype):
    c = TN.Case(tmp_path, ctx, C.config(96, 61, [C.hgrn2(heads, dk, dv), C.gla(heads, dk, dv, ff=64)]), heads + dk + dv)
    n = 400
    toks = TN.tokens(c.cfg, n, 5)
    want = c.want(toks)
    m = c.open(dtype, n)
    states = []
    for cuts in ([n], [17, 1, 33, 130, 3, 216], [99, 101, 200], [16, 2, 128, 129, 125]):
        m.reset_state()
        TN.check(TN.feed(m, toks, cuts), want, dtype, cuts)
        states.append(m.get_state(0, 0, np.float32, heads * dk * dv))
    for s in states[1:]:
        assert np.isfinite(s).all() and np.max(np.abs(s - states[0])) <= (2e-5 if dtype == "float32" else 1e-2) * np.max(np.abs(states[0]))
    assert ctx.device_status() == 0
    m.close()
