"""Kernels of long portions that share out rows: token tiles of the causal convolution with a remainder, norms of a warp a group, narrow products of ragged
sizes, the grouping of more (token, expert) pairs than its threads hold, over several scans of 32 experts, and norms of rows and groups on both sides of what a warp, a
thread's eight values and a CTA's registers hold."""
import numpy as np
import pytest

import test_gpu_netusun as netusun
import test_gpu_rutulix as rutulix
from test_gpu_hybrid import F32_TOL, att_layer, close_bf16, ho, mk, model_cfg, rel, ssd_layer, tokens_for  # noqa: F401
from test_gpu_netusun import no  # noqa: F401
from test_gpu_rutulix import ro  # noqa: F401

mk_netusun, mk_rutulix = netusun.mk, rutulix.mk

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tokens,top,seed", [(603, 6, 5), (1371, 12, 6)])   # 603 rows x 3 groups = 1809 warps; 1371 x 12 pairs = 16 452 (16 x 1024 are held)
def test_long_portion(mk, ho, tokens, top, seed):  # noqa: F811
    cfg = ho.small_config()
    cfg["layers"] = [dict(cfg["layers"][1], mlp={"kind": "moe", "router": {"experts": 41, "top": top, "scale": 1.0}, "expert": {"ff": 16, "limit": 2.0}}),
                     cfg["layers"][0]]
    m, W = mk(cfg, seed=seed, chunk=tokens)
    toks = tokens_for(cfg, tokens, 3)
    exp, exp_layers = ho.run(cfg, W, toks)
    got, got_layers = m.forward_chunk(toks, 0, range(tokens), layers=True)
    assert rel(got_layers, exp_layers) < F32_TOL
    assert rel(got, exp) < F32_TOL


# groups of 1000 and 1024 values, more than the CTAs that the device holds: a warp each; of 1026 and 2048: a CTA each, in registers; of 2050: read twice
@pytest.mark.parametrize("width,groups,tokens", [(3000, 3, 500), (2048, 2, 700), (2052, 2, 620), (4096, 2, 5), (4100, 2, 5)])
def test_norm_groups(mk, ho, width, groups, tokens):  # noqa: F811
    cfg = model_cfg([ssd_layer(heads=2, vdim=6, state=4, groups=1, conv=2, ng=2), att_layer(heads=1, dim=4, vdim=3, rank=5, win=9)], width=width, groups=groups)
    m, W = mk(cfg, seed=7, chunk=tokens)
    toks = tokens_for(cfg, tokens, 4)
    exp, exp_layers = ho.run(cfg, W, toks)
    got, got_layers = m.forward_chunk(toks, 0, range(tokens), layers=True)
    assert rel(got_layers, exp_layers) < F32_TOL
    assert rel(got, exp) < F32_TOL


@pytest.mark.parametrize("width", [2048, 2056, 4096, 4100])   # eight values a thread up to 2048, sixteen up to 4096, norms by themselves behind that
def test_norms_of_closing_blocks(mk_netusun, no, width):  # noqa: F811
    cfg = no.model_config([no.att(heads=2, dim=8, vdim=6, mlp=no.moe(6, 3, 8, 2, 1, 1.0, 11)), no.mem(heads=2, dim=4, vdim=5, mlp=no.dense(12))], width=width, vocab=61)
    m, W = mk_netusun(cfg, seed=3, chunk=24)
    toks = tokens_for(cfg, 21, 5)
    exp = no.run(cfg, W, toks)
    assert rel(m.forward_chunk(toks, 0, range(21)), exp[0] if isinstance(exp, tuple) else exp) < F32_TOL


# ends of column tiles of bf16 products on the tensor cores: last blocks of 4, 8 and 28 columns, of an odd number, tiles of one block and of several for the two warps that share a row
# block's columns; plain, gated, on top of the rows, gates on what lies there
@pytest.mark.parametrize("width,ff,vocab,tokens", [(40, 36, 131, 33), (72, 132, 132, 129), (136, 100, 260, 200), (520, 284, 97, 70)])
def test_ends_of_column_tiles(mk_netusun, no, width, ff, vocab, tokens):  # noqa: F811
    cfg = no.model_config([no.att(heads=3, dim=12, vdim=12, size=40, mlp=no.dense(ff)), no.mem(heads=2, dim=9, vdim=14, mlp=no.moe(5, 2, ff + 4, shared=ff)), no.lat(mlp=no.dense(ff + 1))],
                          width=width, vocab=vocab)
    m, W = mk_netusun(cfg, seed=ff, chunk=256, quant="bf16")
    toks = tokens_for(cfg, tokens, 3)
    assert netusun.close_bf16(m.forward_chunk(toks, 0, range(tokens)), no.run(cfg, W, toks)[0], no.rounding_noise(cfg, W, toks))


@pytest.mark.parametrize("width,ff,tokens", [(40, 36, 45), (72, 260, 130), (136, 1028, 200)])   # xIELU: activations without a branch, rounded as they are stored
def test_activations_of_column_tiles(mk_rutulix, ro, width, ff, tokens):  # noqa: F811
    cfg = ro.model_config([ro.att(ff=ff), ro.att(heads=4, dim=10, ff=ff + 8)], width=width, vocab=131)
    m, W = mk_rutulix(cfg, seed=ff, chunk=256, quant="bf16")
    toks = tokens_for(cfg, tokens, 3)
    assert rutulix.close_bf16(m.forward_chunk(toks, 0, range(tokens)), ro.run(cfg, W, toks)[0])


# a gate whose values are looked up by a row's token, more columns than the narrow products take: rows past the portion's end belong to no token (portions of a few rows, of a tile
# less one, of a row more, smaller than the chunk; fewer tokens in the vocabulary than rows in a chunk)
@pytest.mark.parametrize("width,side,vocab,tokens,chunk", [(40, 104, 31, 40, 60), (64, 100, 53, 5, 8), (72, 256, 53, 127, 200), (40, 128, 97, 129, 129)])
def test_rows_looked_up_by_token(mk, ho, width, side, vocab, tokens, chunk):  # noqa: F811
    cfg = model_cfg([ssd_layer(heads=2, vdim=8, state=8), att_layer()], width=width, vocab=vocab, side=side)
    m, W = mk(cfg, seed=side, chunk=chunk, quant="bf16")
    toks = tokens_for(cfg, tokens, 3)
    assert close_bf16(m.forward_chunk(toks, 0, range(tokens)), ho.run(cfg, W, toks)[0])
