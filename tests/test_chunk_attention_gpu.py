"""GPU: prompt attention on the 5th-generation tensor cores, at head sizes that it takes (whole 64s of key features after padding, 64, 128 or 256 value
features) and at the edges of its tiles: 128 query rows (tokens x heads), 128 keys, ring and buffer turnovers, windows that begin inside a tile of rows or of
keys, sinks, rotated values, a key part shared by all heads, portions down to one token.  Logits against the plain statements in oracle/, with the bounds of the
models' own tests (bf16 operands in the projections), and whole prompt against portions."""
import numpy as np
import pytest

import nufalorn_cases as C
import test_nufalorn_gpu as TN
import test_vobunex_gpu as TV
import vobunex_cases as CV

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("heads,kv,dim,vdim,block,rot", [(4, 2, 64, 64, 100, None), (6, 1, 128, 64, 1000, 16), (3, 3, 128, 128, 128, None), (8, 2, 120, 116, 77, 8),
                                                         (2, 2, 192, 128, 300, 64), (5, 1, 256, 256, 129, 32), (4, 4, 64, 250, 5000, None)])
def test_windows(ctx, lb, tmp_path, heads, kv, dim, vdim, block, rot):
    c = TN.Case(tmp_path, ctx, C.config(96, 89, [C.att(heads, kv, dim, vdim, block, rot_dims=rot, ff=64), C.att(heads, kv, dim, vdim, block + 50, rot_dims=rot)]), 31)
    n = 420
    toks = TN.tokens(c.cfg, n, 3)
    want = c.want(toks)
    m = c.open("bfloat16", n)
    for cuts in ([n], [127, 1, 128, 2, 130, 32], [33, 95, 129, 163], [1, 255, 164]):
        m.reset_state()
        TN.check(TN.feed(m, toks, cuts), want, "bfloat16", cuts)
    assert ctx.device_status() == 0
    m.close()


@pytest.mark.parametrize("heads,dim,rot,vdim", [(3, 64, 64, 64), (5, 128, 64, 128), (2, 128, 128, 60)])
def test_shared_key_part(ctx, lb, tmp_path, heads, dim, rot, vdim):
    c = TV.Case(tmp_path, ctx, CV.config(72, 83, [CV.latent(heads, dim, rot, vdim, 48, 64), CV.latent(heads, dim, rot, vdim, 48, 64)]), 17)
    n = 300
    toks = TV.tokens(c.cfg, n, 5)
    want = c.want(toks)
    m = c.open("bfloat16", n)
    for cuts in ([n], [16, 112, 129, 43], [255, 45]):
        m.reset_state()
        TV.check(TV.feed(m, toks, cuts), want, "bfloat16", cuts)
    assert ctx.device_status() == 0
    m.close()


@pytest.mark.parametrize("block", [700, 5000])
def test_few_rows_behind_many_keys(ctx, lb, tmp_path, block):
    """the keys of a tile of rows dealt to several CTAs: parts of unequal length, parts without visible keys (a window that begins far along)"""
    c = TN.Case(tmp_path, ctx, C.config(96, 89, [C.att(4, 2, 128, 128, block, rot_dims=32), C.att(6, 2, 64, 64, block)]), 33)
    n = 1500
    toks = TN.tokens(c.cfg, n, 4)
    want = c.want(toks)
    m = c.open("bfloat16", n)
    for cuts in ([1400, 2, 5, 33, 60], [695, 8, 300, 129, 368]):
        m.reset_state()
        TN.check(TN.feed(m, toks, cuts), want, "bfloat16", cuts)
    assert ctx.device_status() == 0
    m.close()


def test_hybrid_few_rows_behind_many_keys(ctx, lb):
    """the same for the int4 hybrid: portions of 1 to 40 tokens behind 900 give the logits of one prompt to the prompt's own tolerance (fp16 activations: 2e-3)"""
    from lithos_b200 import model as M
    cfg = M.tiny(max_ctx=1024)
    m = M.Model(ctx, cfg)
    m.fill_synthetic(9)
    toks = np.random.default_rng(5).integers(0, cfg.vocab, 960).tolist()
    want = m.forward(toks, 0, list(range(900, 960)))
    m.reset_state()
    m.forward(toks[:900], 0, [])
    got, pos = [], 900
    for n in (5, 2, 40, 13):
        got.append(m.forward(toks[pos:pos + n], pos, list(range(n))))
        pos += n
    got = np.concatenate(got)
    assert ctx.device_status() == 0
    assert np.max(np.abs(got - want)) <= 4e-3 * np.max(np.abs(want))
    m.close()
