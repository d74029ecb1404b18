"""Portions through attention with mixed heads, against the float64 statement: the mixing and softmax kernel with its scores in registers (up to 16
and up to 32 heads) and in shared memory (more), the mixed scores kept on chip and, where heads x keys are too many, in place; blocks of 512
queries, and score and value products that leave out what a block of queries does not see (chunk mask: keys of earlier chunks)."""
import pytest

from test_gpu_rutulix import F32_TOL, mk, peaky, rel, ro, tokens_for  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("heads,kv_heads,size,tokens", [(3, 1, 500, 90), (16, 4, 700, 640), (17, 17, 40, 600), (64, 4, 700, 640), (32, 2, 400, 390)])
def test_one_portion(mk, ro, heads, kv_heads, size, tokens):  # noqa: F811
    cfg = ro.model_config([ro.att(heads=heads, kv_heads=kv_heads, dim=8, size=size)], width=48)
    m, W = mk(cfg, seed=heads, chunk=tokens, edit=peaky)
    toks = tokens_for(cfg, tokens, 7)
    rows = sorted({0, 1, 63, 64, size - 1, size, 511, 512, tokens - 1} & set(range(tokens)))
    assert rel(m.forward_chunk(toks, 0, rows), ro.run(cfg, W, toks)[0][rows]) < F32_TOL
