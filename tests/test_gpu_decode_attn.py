"""Attention of decode-sized steps where its split of heads, tokens, depth and value columns can go wrong, against the float64 statement:
more than 8 query heads per key head, depths that are not a multiple of 4, one to four value columns per thread, shares of the keys, and
steps of 1 to 31 tokens (the CTA holds heads of one token, or neighbouring tokens of one head)."""
import pytest

from test_gpu_netusun import F32_TOL, in_portions, mk, no, rel, tokens_for  # noqa: F401

pytestmark = pytest.mark.gpu

PORTIONS = [[], [2] * 30, [3] * 20, [5] * 12, [9, 17, 31]]   # [] decodes token by token


@pytest.mark.parametrize("heads,kv_heads,dim,vdim", [(12, 1, 10, 6), (9, 3, 96, 260), (4, 4, 33, 5), (20, 2, 4, 600)])
def test_grouped_heads(mk, no, heads, kv_heads, dim, vdim):  # noqa: F811
    cfg = no.model_config([no.att(heads=heads, kv_heads=kv_heads, dim=dim, vdim=vdim, size=45), no.att(heads=heads, kv_heads=kv_heads, dim=dim, vdim=vdim, size=None)], width=48, vocab=97)
    m, W = mk(cfg, seed=heads + dim, chunk=31)
    toks = tokens_for(cfg, 70, 6)
    exp = no.run(cfg, W, toks)[0]
    for sizes in PORTIONS:
        assert rel(in_portions(m, toks, sizes), exp) < F32_TOL


@pytest.mark.parametrize("heads,kv_rank,rot_dim", [(3, 13, 4), (10, 250, 8), (9, 300, 6), (2, 700, 4)])
def test_latents(mk, no, heads, kv_rank, rot_dim):  # noqa: F811
    cfg = no.model_config([no.lat(heads=heads, kv_rank=kv_rank, rot_dim=rot_dim)], width=40, vocab=97)
    m, W = mk(cfg, seed=kv_rank, chunk=31)
    toks = tokens_for(cfg, 70, 7)
    exp = no.run(cfg, W, toks)[0]
    for sizes in PORTIONS:
        assert rel(in_portions(m, toks, sizes), exp) < F32_TOL


@pytest.mark.parametrize("heads,kv_heads", [(16, 16), (8, 4), (5, 5)])
def test_shares_of_several_tiles(mk, no, heads, kv_heads):  # noqa: F811
    """Windows so wide, over so many key heads, that a CTA's share of the keys is more than a tile: 72 tiles and more in shares of up to 3, 2 and 2."""
    cfg = no.model_config([no.att(heads=heads, kv_heads=kv_heads, dim=16, vdim=12, size=None)] * 2, width=48, vocab=97)
    m, W = mk(cfg, seed=heads, chunk=200, context=2300)
    toks = tokens_for(cfg, 240, 6)
    exp = no.run(cfg, W, toks)[0]
    for sizes in ([], [200, 2, 2, 3, 3, 4, 4], [90, 1, 4, 3, 2, 100]):
        assert rel(in_portions(m, toks, sizes), exp) < F32_TOL
