"""GPU: a prompt's products on CTA pairs (tiles of 256 weight rows x 256 tokens) and on single CTAs.

* A prompt whose input products take pairs by themselves: two matrices in one launch, a last pair tile with rows for one CTA only, a ragged token tile,
  and as many tiles as make accumulators alternate; against oracle/nufalorn.py, tolerances as in test_nufalorn_gpu.py (bf16 operands).
* Every product of both kinds of models on pairs (tiles with rows for one CTA only, token tiles down to one token, every epilogue) and none:
  a product's sums run over k in the same order either way, so the logits are the same bits.
"""
import numpy as np
import pytest

import nufalorn_cases as C
import vobunex_cases as V
from oracle import nufalorn as N

pytestmark = pytest.mark.gpu


def forward(ctx, m, toks, rows, mode):
    """logits of a prompt with the products on pairs by rule (1), never (0) or always (2), and how many ran so"""
    ctx.set_product_pairs(mode)
    try:
        m.reset_state()
        got = np.asarray(m.forward(toks, 0, rows))
    finally:
        n = ctx.set_product_pairs(1)
    assert ctx.device_status() == 0 and np.isfinite(got).all()
    return got, n


@pytest.mark.parametrize("T", [1000, 897])
def test_pair_products(ctx, tmp_path, T):
    from lithos_b200 import model as M
    cfg = C.config(4096, 48, [C.att(3, 1, 64, 64, 512, ff=8256)])
    w = C.tensors(cfg, 3)
    toks = np.random.default_rng(T).integers(0, cfg["vocab"], T).tolist()
    m = M.Model.open(ctx, C.write(tmp_path, cfg, w), 1024, "bfloat16")
    got, n = forward(ctx, m, toks, list(range(T)), 1)
    assert n > 0
    single, n = forward(ctx, m, toks, list(range(T)), 0)
    assert n == 0 and np.array_equal(got, single)
    m.close()
    want = N.Nufalorn(cfg, w).run(toks)
    e = np.sqrt(np.mean((np.asarray(got, np.float64) - want) ** 2, axis=-1)) / np.sqrt(np.mean(want ** 2))
    assert np.isfinite(e).all() and e.max() <= 4e-2 and e.mean() <= 1.5e-2, (int(e.argmax()), e.max(), e.mean())


@pytest.mark.parametrize("T", [40, 257, 700])
@pytest.mark.parametrize("kind", ["nufalorn", "vobunex"])
def test_all_products_on_pairs(ctx, tmp_path, kind, T):
    from lithos_b200 import model as M
    if kind == "nufalorn":
        cfg = C.config(256, 48, [C.att(3, 1, 64, 64, 128, ff=320), C.hgrn2(2, 64, 64), C.gla(2, 64, 64, ff=192), C.att(2, 2, 64, 64, 128)])
        w = C.tensors(cfg, 4)
    else:
        cfg = V.config(256, 48, [V.latent(3, 20, 8, 36, 24, 40, mlp=V.dense(300)), V.mamba2(4, 18, 24, groups=2, mlp=V.moe(24, 4, 2)), V.mamba2(2, 16, 16, mlp=V.dense(72))])
        w = V.tensors(cfg, 4)
    toks = np.random.default_rng(T).integers(0, cfg["vocab"], T).tolist()
    m = M.Model.open(ctx, (C if kind == "nufalorn" else V).write(tmp_path, cfg, w), 1024, "bfloat16")
    rows = list(range(0, T, 7)) + [T - 1]
    pairs, n = forward(ctx, m, toks, rows, 2)
    assert n > 0
    single, n = forward(ctx, m, toks, rows, 0)
    m.close()
    assert n == 0 and np.array_equal(pairs, single)
