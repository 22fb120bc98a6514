"""GPU: a prompt whose products run on CTA pairs (tiles of 256 weight rows x 256 tokens): two matrices in one launch, a last pair tile with rows for one
CTA only, a ragged token tile, every epilogue of a parallel layer, and as many tiles as make accumulators alternate, against oracle/nufalorn.py.

Tolerances as in test_nufalorn_gpu.py (bf16 operands)."""
import numpy as np
import pytest

import nufalorn_cases as C
from oracle import nufalorn as N

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T", [1000, 897])
def test_pair_products(ctx, tmp_path, T):
    from lithos_b200 import model as M
    cfg = C.config(2048, 48, [C.att(3, 1, 64, 64, 512, ff=8256)])
    w = C.tensors(cfg, 3)
    toks = np.random.default_rng(T).integers(0, cfg["vocab"], T).tolist()
    m = M.Model.open(ctx, C.write(tmp_path, cfg, w), 1024, "bfloat16")
    got = m.forward(toks, 0, list(range(T)))
    assert ctx.device_status() == 0
    m.close()
    want = N.Nufalorn(cfg, w).run(toks)
    e = np.sqrt(np.mean((np.asarray(got, np.float64) - want) ** 2, axis=-1)) / np.sqrt(np.mean(want ** 2))
    assert np.isfinite(e).all() and e.max() <= 4e-2 and e.mean() <= 1.5e-2, (int(e.argmax()), e.max(), e.mean())
