"""GPU: prompts whose products add to the residual or apply SwiGLU themselves (from 33 tokens on), at the token counts where those products change and around
them, against the same tokens in portions of at most 32, which take the separate kernels: logits and, in the tokens that follow, states and caches agree to the
prompt pass's tolerance (fp16 activations: 2e-3 of the largest logit, twice that for two runs that both differ from the exact value)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [33, 48, 64, 65, 128, 129, 160, 161, 177, 256, 257, 300])
def test_epilogues(ctx, lb, n):
    from lithos_b200 import model as M
    cfg = M.tiny(max_ctx=384)
    m = M.Model(ctx, cfg)
    m.fill_synthetic(n)
    toks = np.random.default_rng(n).integers(0, cfg.vocab, n + 4).tolist()
    got = []
    for step in (n, 32):
        m.reset_state()
        for pos in range(0, n, step):
            last = m.forward(toks[pos:min(n, pos + step)], pos, [min(n, pos + step) - pos - 1])
        got.append([last] + [m.forward(toks[n + i:n + i + 1], n + i, [0]) for i in range(4)])
    assert ctx.device_status() == 0
    for a, b in zip(*got):
        assert np.max(np.abs(a - b)) <= 4e-3 * np.max(np.abs(b))
    m.close()
