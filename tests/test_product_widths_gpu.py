"""GPU: token tiles of a prompt's products in steps of 16 between the powers of two: 132 row tiles at token counts whose best width is such a one, ragged last
tiles; against oracle/nufalorn.py, tolerances as in test_nufalorn_gpu.py (bf16 operands)."""
import numpy as np
import pytest

import nufalorn_cases as C
import test_nufalorn_gpu as TN

pytestmark = pytest.mark.gpu


def test_widths_between(ctx, lb, tmp_path):
    c = TN.Case(tmp_path, ctx, C.config(1024, 48, [C.att(3, 1, 64, 64, 512, ff=8256)]), 7)
    toks = TN.tokens(c.cfg, 470, 2)
    want = c.want(toks)
    m = c.open("bfloat16", 512)
    for T in (130, 145, 200, 330, 470):
        m.reset_state()
        TN.check(np.asarray(m.forward(toks[:T], 0, list(range(T)))), want[:T], "bfloat16", T)
    assert ctx.device_status() == 0
    m.close()
