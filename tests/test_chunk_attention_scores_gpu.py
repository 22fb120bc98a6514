"""GPU: prompt attention of the int4 hybrid with scores far below zero: norms of queries and keys so large that scores reach 1e33, where a row that sees negative
ones only (the first token's, in about half of the heads) has a largest score below -1e30; its weights still add up to one.  Logits against the CPU oracle decoding the same
tokens one by one, tolerance as in test_prefill_gpu.py.

Such a softmax picks one row, and the two sides' scores differ by the projections' fp16 activations (2^-11 each, about 5e-4 of a score): two largest scores closer
than that may be picked by either side (a few in a thousand rows that see many).  So prompts of up to five tokens are compared, a longer one has to be finite."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 5, 40])
def test_scores_far_below_zero(ctx, lb, oracle, n):
    from lithos_b200 import model as M
    cfg = M.tiny(max_ctx=96)
    slots = [M.synthetic_layer_slots(cfg, 11, l) for l in range(cfg.n_layers)]
    glob = M.synthetic_globals(cfg, 11)
    for l in range(cfg.n_layers):
        if cfg.is_fa(l):
            for name in ("FA_Q_NORM", "FA_K_NORM"):
                w = lb.bf16_to_f32(slots[l][M.WS[name]])
                slots[l][M.WS[name]] = lb.f32_to_bf16((w * 2.0 ** 55).astype(np.float32))
    om = oracle.Model(oracle.ModelCfg(**{k: getattr(cfg, k) for k, _ in M.ModelCfg._fields_}), slots, glob)
    gm = M.Model(ctx, cfg)
    for l in range(cfg.n_layers):
        gm.load_layer(l, slots[l])
    gm.load_globals(glob)
    toks = np.random.default_rng(n).integers(0, cfg.vocab, n).tolist()
    want = []
    for pos, tok in enumerate(toks):
        om.decode(tok, pos)
        want.append(om.logits().copy())
    got = np.asarray(gm.forward(toks, 0, list(range(n))))
    want = np.asarray(want)
    assert ctx.device_status() == 0 and np.isfinite(got).all()
    assert n > 5 or np.max(np.abs(got - want)) <= 2e-3 * np.max(np.abs(want))
    gm.close()
    om.close()
