"""bf16 products of portions on the tensor cores, at the edges of their tiles (128 rows; 32 to 256 columns; 64-deep slices; experts with
no row, one tile and several), against the float64 statement of a small model made of them."""
import numpy as np
import pytest

from test_gpu_netusun import close_bf16, mk, no, tokens_for  # noqa: F401
from test_gpu_zetivik import mk as mk_zetivik  # noqa: F401
from test_gpu_zetivik import zo  # noqa: F401

pytestmark = pytest.mark.gpu


# width: depth of most products (72 and 136 end inside a 64-deep slice), ff: their columns (104 and 264 end inside a column tile; gated ones take
# half a tile), tokens: rows (5 is the smallest portion that takes this path; 128 is one row tile)
@pytest.mark.parametrize("width,ff,tokens", [(72, 104, 5), (136, 264, 127), (128, 256, 128), (64, 1032, 129), (136, 104, 257)])
def test_dense_edges(mk, no, width, ff, tokens):  # noqa: F811
    cfg = no.model_config([no.att(heads=4, dim=32, vdim=24, size=40, mlp=no.dense(ff)), no.lat(mlp=no.dense(2 * ff))], width=width, vocab=211)
    m, W = mk(cfg, seed=width + tokens, quant="bf16", chunk=512)
    toks = tokens_for(cfg, tokens, 3)
    assert close_bf16(m.forward_chunk(toks, 0, range(tokens)), no.run(cfg, W, toks)[0], no.rounding_noise(cfg, W, toks))


@pytest.mark.parametrize("experts,top,ff,tokens", [(3, 1, 40, 5), (2, 2, 72, 130), (8, 2, 104, 200), (40, 3, 8, 64)])
def test_routed_edges(mk, no, experts, top, ff, tokens):  # noqa: F811
    cfg = no.model_config([no.att(heads=2, dim=16, vdim=16, mlp=no.moe(experts=experts, top=top, ff=ff, shared=ff + 32))], width=88, vocab=131)
    m, W = mk(cfg, seed=experts, quant="bf16", chunk=256)
    toks = tokens_for(cfg, tokens, 4)
    assert close_bf16(m.forward_chunk(toks, 0, range(tokens)), no.run(cfg, W, toks)[0], no.rounding_noise(cfg, W, toks))


# results stored by rows (32 bytes a lane) and turned through shared memory: rows of C that are no multiple of eight columns (84), blocks of 32
# columns that end inside the matrix (72, 136, 264), whole ones (256); additions into the residual rows, gated pairs, scattered expert rows
@pytest.mark.parametrize("width,experts,top,ff,tokens", [(84, 2, 1, 104, 60), (136, 2, 2, 264, 256), (256, 3, 2, 128, 300), (100, 1, 1, 72, 129)])
def test_stores(mk, no, width, experts, top, ff, tokens):  # noqa: F811
    cfg = no.model_config([no.att(heads=4, dim=32, vdim=24, size=40, mlp=no.moe(experts=experts, top=top, ff=ff, shared=2 * ff)), no.lat(mlp=no.dense(ff))],
                          width=width, vocab=131)
    m, W = mk(cfg, seed=tokens, quant="bf16", chunk=512)
    toks = tokens_for(cfg, tokens, 6)
    assert close_bf16(m.forward_chunk(toks, 0, range(tokens)), no.run(cfg, W, toks)[0], no.rounding_noise(cfg, W, toks))


def test_unaligned_depth_and_short_steps(mk, no):  # noqa: F811
    """Depths that TMA cannot address (not a multiple of 8) and the steps of up to four rows keep their own kernels."""
    cfg = no.model_config([no.att(heads=3, dim=10, vdim=6, mlp=no.dense(98))], width=84, vocab=61)
    m, W = mk(cfg, seed=9, quant="bf16", chunk=64)
    toks = tokens_for(cfg, 40, 5)
    exp, noise = no.run(cfg, W, toks)[0], no.rounding_noise(cfg, W, toks)
    assert close_bf16(m.forward_chunk(toks, 0, range(40)), exp, noise)
    rows = np.concatenate([m.forward_chunk(toks[p:p + 4], p, range(4)) for p in range(0, 40, 4)])
    assert close_bf16(rows, exp, noise)


# More than three tiles of 128 x 256 per CTA (148 of them), so that both accumulators go round, the ring's indices run on over tiles and what a tile adds to is
# fetched under the products of the one ahead.  1024 rows are 8 row tiles.  Stored: 57 column tiles; added: the same onto the stream; gated: tiles of
# 128 columns, 57 of them; routed: some 18 row tiles by 29 column tiles
@pytest.mark.parametrize("kind", ["stored", "gated", "routed"])
def test_many_tiles_per_cta(mk, no, kind):  # noqa: F811
    wide, att = 14344, dict(heads=2, dim=16, vdim=8, size=9)
    if kind == "stored":
        cfg = no.model_config([no.att(**att)], width=wide, vocab=131)
    else:
        cfg = no.model_config([no.att(mlp=no.dense(7208) if kind == "gated" else no.moe(experts=3, top=2, ff=3656, shared=None), **att)], width=104, vocab=131)
    m, W = mk(cfg, seed=len(kind), quant="bf16", chunk=1024, context=1100)
    toks = tokens_for(cfg, 1024, 7)
    assert close_bf16(m.forward_chunk(toks, 0, range(1024)), no.run(cfg, W, toks)[0], no.rounding_noise(cfg, W, toks))


def test_many_tiles_added(mk_zetivik, zo):  # noqa: F811
    cfg = zo.model_config([zo.light(heads=3, dim=8, vdim=8, ff=16)], width=14344, vocab=131)
    m, W = mk_zetivik(cfg, seed=5, quant="bf16", chunk=1024, context=1100)
    toks = tokens_for(cfg, 1024, 7)
    assert close_bf16(m.forward_chunk(toks, 0, range(1024)), zo.run(cfg, W, toks)[0], zo.rounding_noise(cfg, W, toks))
