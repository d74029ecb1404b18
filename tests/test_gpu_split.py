"""fp32 products of portions in three bf16 parts on the tensor cores, at the edges of their tiles (128 rows, split 64 at a time; 64 columns, gated ones 32; 64-deep slices in
halves of 32, three of them in the ring), against the float64 statement of a small model made of them."""
import numpy as np
import pytest

from test_gpu_netusun import F32_TOL, in_portions, mk, no, rel, tokens_for  # noqa: F401

pytestmark = pytest.mark.gpu


# width: depth of most products (36 and 68 end inside a half slice, 66 and 133 have rows that take no 16-byte loads, 772 and 1028 go round the ring several times),
# ff: columns (gated) and depth of the second product, tokens: rows
@pytest.mark.parametrize("width,ff,tokens", [(36, 20, 5), (64, 32, 63), (66, 33, 64), (68, 97, 65), (133, 130, 127), (260, 64, 128), (772, 200, 129), (1028, 36, 193)])
def test_dense_edges(mk, no, width, ff, tokens):  # noqa: F811
    cfg = no.model_config([no.att(heads=3, dim=20, vdim=12, size=40, mlp=no.dense(ff)), no.lat(mlp=no.dense(2 * ff))], width=width, vocab=131)
    m, W = mk(cfg, seed=width + tokens, chunk=256)
    toks = tokens_for(cfg, tokens, 3)
    assert rel(m.forward_chunk(toks, 0, range(tokens)), no.run(cfg, W, toks)[0]) < F32_TOL


# experts with no row, some, one tile and more; the second step's products read rows of the first in other orders
@pytest.mark.parametrize("experts,top,ff,sizes", [(3, 1, 40, [5, 60]), (2, 2, 72, [130]), (40, 3, 9, [64, 65]), (5, 2, 260, [200])])
def test_routed_edges(mk, no, experts, top, ff, sizes):  # noqa: F811
    cfg = no.model_config([no.att(heads=2, dim=16, vdim=16, mlp=no.moe(experts=experts, top=top, ff=ff, shared=ff + 31))], width=88, vocab=131)
    m, W = mk(cfg, seed=experts, chunk=256)
    toks = tokens_for(cfg, sum(sizes), 4)
    assert rel(in_portions(m, toks, sizes), no.run(cfg, W, toks)[0]) < F32_TOL


# tiles whose depth two, four or eight CTAs share: ragged last slices, shares without a slice (17 slices over 8 CTAs: the last one has two, 9 over 8: three have none), narrow router products
@pytest.mark.parametrize("width,ff,tokens", [(520, 40, 40), (1100, 36, 70), (2060, 24, 5), (2048, 16, 460), (600, 700, 130)])
def test_shared_depth(mk, no, width, ff, tokens):  # noqa: F811
    cfg = no.model_config([no.att(heads=2, dim=16, vdim=16, mlp=no.moe(experts=6, top=2, ff=ff, shared=ff))], width=width, vocab=67)
    m, W = mk(cfg, seed=width, chunk=512)
    toks = tokens_for(cfg, tokens, 4)
    assert rel(m.forward_chunk(toks, 0, range(tokens)), no.run(cfg, W, toks)[0]) < F32_TOL


# Products of few slices, positive operands: the tensor core truncates its additions, so that results are too small on average, by 4.1e-8 with additions of 16 values joined in registers, by
# 3.5e-8 with accumulators of 32 values, by 7e-8 with accumulators of 64.  (The norm ahead of the product has errors of either sign, one a row.)
@pytest.mark.parametrize("width", [48, 64, 128, 200, 320])
def test_truncation_of_few_slices(mk, no, width):  # noqa: F811
    def edit(W):
        W["embed"], W["final.norm"] = np.abs(W["embed"]), np.abs(W["final.norm"])
        W["l0.mix.o"] = W["l0.mix.o"] * 0.0                  # the stream is the embedding
    cfg = no.model_config([no.att(heads=1, dim=16, vdim=16, mlp=None)], width=width, vocab=500)
    m, W = mk(cfg, seed=width, chunk=512, edit=edit)
    toks = tokens_for(cfg, 500, 3)
    got, exp = m.forward_chunk(toks, 0, range(500)), no.run(cfg, W, toks)[0]
    assert np.all(exp > 0) and abs(float(np.mean(got.astype(np.float64) / exp - 1.0))) < 5e-8
