"""Attention of portions in one kernel at the edges of its tiles (16 query rows a warp, 32 keys, depths padded to 16, value columns in groups of 64
or 128), against the float64 statement: steps that continue a sequence inside a window, several column groups, heads too deep for the kernel."""
import pytest

from test_gpu_hybrid import close_bf16 as close_rows
from test_gpu_hybrid import ho  # noqa: F401
from test_gpu_hybrid import mk as mk_hybrid  # noqa: F401
from test_gpu_netusun import F32_TOL, close_bf16, in_portions, mk, no, rel, tokens_for  # noqa: F401
from test_gpu_sakusun import mk as mk_sakusun  # noqa: F401
from test_gpu_sakusun import so  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("heads,kv_heads,dim,vdim,size", [(3, 1, 10, 6, 1), (4, 2, 33, 65, 40), (2, 2, 128, 128, 33), (6, 3, 16, 300, None), (1, 1, 300, 20, 50)])
def test_grouped_heads(mk, no, heads, kv_heads, dim, vdim, size):  # noqa: F811
    cfg = no.model_config([no.att(heads=heads, kv_heads=kv_heads, dim=dim, vdim=vdim, size=size)] * 2, width=48, vocab=97)
    m, W = mk(cfg, seed=heads + dim, chunk=160)
    toks = tokens_for(cfg, 210, 8)
    exp = no.run(cfg, W, toks)[0]
    for sizes in ([160, 50], [33, 32, 129], [32, 160]):
        assert rel(in_portions(m, toks, sizes), exp) < F32_TOL


@pytest.mark.parametrize("heads,dim,rot_dim,vdim", [(3, 7, 4, 5), (2, 128, 64, 128), (2, 40, 8, 129)])
def test_latents(mk, no, heads, dim, rot_dim, vdim):  # noqa: F811
    cfg = no.model_config([no.lat(heads=heads, dim=dim, rot_dim=rot_dim, vdim=vdim)], width=40, vocab=97)
    toks = tokens_for(cfg, 200, 9)
    for quant in ("fp32", "bf16"):
        m, W = mk(cfg, seed=dim, chunk=128, quant=quant)
        exp = no.run(cfg, W, toks)[0]
        noise = no.rounding_noise(cfg, W, toks) if quant == "bf16" else None
        for sizes in ([128, 72], [33, 95, 65]):
            got = in_portions(m, toks, sizes)
            assert rel(got, exp) < F32_TOL if quant == "fp32" else close_bf16(got, exp, noise)


@pytest.mark.parametrize("size,keep", [(20, 3), (70, 40), (1, 1), (20, 0)])
def test_kept_positions_of_deep_heads(mk_sakusun, so, size, keep):  # noqa: F811
    """Heads too deep for the one kernel (335 is the deepest): score and value products that leave out what a block of queries does not see.  Kept
    first positions stay visible to queries whose window has left them behind, also where the step's range starts with them."""
    cfg = so.model_config([so.att(heads=2, kv_heads=1, dim=352, vdim=20, size=size, keep_first=keep, scale=0.05, ff=None)], width=48, vocab=97)
    m, W = mk_sakusun(cfg, seed=size, chunk=300)
    toks = tokens_for(cfg, 360, 8)
    exp = so.run(cfg, W, toks)[0]
    for sizes in ([300, 60], [33, 40, 287]):
        assert rel(in_portions(m, toks, sizes), exp) < F32_TOL


def test_last_block_of_one_query(mk_sakusun, so):  # noqa: F811
    """Blocks of 256 queries whose last one is a single row: its products read keys and values that were packed a launch ahead."""
    cfg = so.model_config([so.att(heads=2, kv_heads=1, dim=352, vdim=20, size=150, keep_first=2, scale=0.05, ff=None)], width=48, vocab=97)
    m, W = mk_sakusun(cfg, seed=2, chunk=300)
    toks = tokens_for(cfg, 290, 8)
    assert rel(in_portions(m, toks, [257, 33]), so.run(cfg, W, toks)[0]) < F32_TOL


# Steps whose query blocks are fewer than the SMs: the keys behind them in shares (of at least four tiles of 32 or 16), joined afterwards; windows that
# cut the shares, several column groups, a depth that takes tiles of 16, kept positions, sinks, a cap and distance biases, gates
@pytest.mark.parametrize("heads,kv_heads,dim,vdim,size", [(2, 1, 12, 10, None), (3, 3, 64, 150, 300), (1, 1, 320, 24, None), (5, 5, 16, 64, 130)])
def test_shares_of_the_keys(mk, no, heads, kv_heads, dim, vdim, size):  # noqa: F811
    cfg = no.model_config([no.att(heads=heads, kv_heads=kv_heads, dim=dim, vdim=vdim, size=size)] * 2, width=48, vocab=97)
    m, W = mk(cfg, seed=heads + dim, chunk=400, context=1200)
    toks = tokens_for(cfg, 1000, 8)
    exp = no.run(cfg, W, toks)[0]
    for sizes in ([400, 400, 200], [399, 33, 100, 32, 130, 306]):
        assert rel(in_portions(m, toks, sizes), exp) < F32_TOL


def test_shares_of_latents(mk, no):  # noqa: F811
    cfg = no.model_config([no.lat(heads=3, dim=40, rot_dim=8, vdim=129), no.lat(heads=2, dim=16, vdim=16)], width=40, vocab=97)
    toks = tokens_for(cfg, 800, 9)
    for quant in ("fp32", "bf16"):
        m, W = mk(cfg, seed=3, chunk=400, quant=quant, context=900)
        exp = no.run(cfg, W, toks)[0]
        got = in_portions(m, toks, [350, 40, 400, 10])
        assert rel(got, exp) < F32_TOL if quant == "fp32" else close_bf16(got, exp, no.rounding_noise(cfg, W, toks))


def test_shares_with_kept_positions(mk_sakusun, so):  # noqa: F811
    cfg = so.model_config([so.att(heads=4, kv_heads=2, dim=8, vdim=8, size=450, keep_first=70, bias_max=200, rel_rows=12, ff=12),
                           so.att(heads=2, dim=8, vdim=70, size=None, softcap=None, v_mix=False, ff=None)], width=40, vocab=97)
    m, W = mk_sakusun(cfg, seed=3, chunk=256, context=1000)
    toks = tokens_for(cfg, 900, 8)
    exp = so.run(cfg, W, toks)[0]
    for sizes in ([256, 256, 256, 132], [250, 250, 40, 33, 256]):
        assert rel(in_portions(m, toks, sizes), exp) < F32_TOL


# heads of 64 entries and more: blocks of 128 queries, tiles of 32 keys, depth in pieces of 64 (65 and 100 end inside one), columns of values in blocks of 64 and 128 (150: two CTAs),
# windows that begin inside a tile, more tiles than a turn of the ring, and shares of the keys (one block of queries behind many keys)
@pytest.mark.parametrize("heads,kv_heads,dim,vdim,size,sizes", [(2, 1, 64, 64, 50, [127, 33]), (3, 3, 65, 70, None, [128, 129]), (4, 2, 128, 128, 200, [300]), (2, 2, 100, 150, 33, [257]),
                                                               (2, 1, 192, 128, None, [130, 126]), (1, 1, 180, 20, 150, [600, 40]), (1, 1, 64, 128, None, [900, 35, 33])])
def test_blocks_of_128_queries(mk, no, heads, kv_heads, dim, vdim, size, sizes):  # noqa: F811
    cfg = no.model_config([no.att(heads=heads, kv_heads=kv_heads, dim=dim, vdim=vdim, size=size)] * 2, width=48, vocab=97)
    m, W = mk(cfg, seed=dim, chunk=1024, context=1100)
    toks = tokens_for(cfg, sum(sizes), 5)
    assert rel(in_portions(m, toks, sizes), no.run(cfg, W, toks)[0]) < F32_TOL


@pytest.mark.parametrize("dim,rot_dim,vdim,tokens", [(64, 64, 64, 150), (128, 64, 128, 260), (72, 8, 129, 140)])
def test_blocks_of_128_queries_with_a_rotated_part(mk, no, dim, rot_dim, vdim, tokens):  # noqa: F811
    cfg = no.model_config([no.lat(heads=2, dim=dim, rot_dim=rot_dim, vdim=vdim)], width=40, vocab=97)
    m, W = mk(cfg, seed=dim, chunk=512, context=600)
    toks = tokens_for(cfg, tokens, 6)
    assert rel(m.forward_chunk(toks, 0, range(tokens)), no.run(cfg, W, toks)[0]) < F32_TOL


# latent attention of bf16 models, operands in one part: blocks of 64 and 128 value columns, depths that end inside a piece of 64, windows inside and over a tile, shares of the keys
@pytest.mark.parametrize("dim,vdim,size,sizes", [(64, 64, 50, [127, 33]), (65, 70, 300, [128, 129]), (128, 128, 200, [300]), (100, 150, 33, [257]), (192, 20, 1000, [130, 126]), (64, 128, 1000, [600, 40])])
def test_blocks_of_128_queries_in_one_part(mk_hybrid, ho, dim, vdim, size, sizes):  # noqa: F811
    att = {"type": "latent_attention", "mixer": {"heads": 2, "dim": dim, "vdim": vdim, "kv_rank": 48, "mask": {"size": size}, "scale": dim ** -0.5}, "mlp": None}
    cfg = ho.small_config(layers=[att] * 2, width=48, norm={"eps": 1e-5, "groups": 1})
    m, W = mk_hybrid(cfg, seed=dim, quant="bf16", chunk=640, context=700)
    toks = tokens_for(cfg, sum(sizes), 5)
    assert close_rows(in_portions(m, toks, sizes), ho.run(cfg, W, toks)[0])
