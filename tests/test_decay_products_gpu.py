"""GPU: decays and betas of hybrid prompts on the tensor cores: both block shapes (48 heads: 8 rows up to 192 tokens, 24 rows from there on), token tiles with 1 to 16 tokens,
a hidden size that is no whole turn of the eight warps, head counts whose rows end inside a tile, the convolution's last inputs behind every portion.  One prompt against
portions of it: logits to the prompt's own tolerance (fp16 activations: 2e-3 each)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("hidden,v_heads,k_heads", [(640, 48, 16), (1024, 6, 2), (1152, 20, 10), (384, 50, 25)])
def test_portions(ctx, lb, hidden, v_heads, k_heads):
    from lithos_b200 import model as M
    cfg = M.tiny(max_ctx=512)
    cfg.hidden, cfg.dn_v_heads, cfg.dn_k_heads = hidden, v_heads, k_heads
    m = M.Model(ctx, cfg)
    m.fill_synthetic(5)
    toks = np.random.default_rng(3).integers(0, cfg.vocab, 480).tolist()
    want = m.forward(toks, 0, list(range(0, 480, 7)))
    for cuts in ([256, 224], [17, 1, 3, 208, 15, 192, 44], [2, 97, 125, 256]):
        assert sum(cuts) == 480
        m.reset_state()
        got, pos = [], 0
        for n in cuts:
            rows = [r - pos for r in range(0, 480, 7) if pos <= r < pos + n]
            y = m.forward(toks[pos:pos + n], pos, rows)
            if rows:
                got.append(y)
            pos += n
        got = np.concatenate(got)
        assert np.isfinite(got).all() and np.max(np.abs(got - want)) <= 4e-3 * np.max(np.abs(want)), cuts
    assert ctx.device_status() == 0
    m.close()
