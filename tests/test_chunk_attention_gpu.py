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
