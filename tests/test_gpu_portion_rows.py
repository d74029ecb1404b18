"""Kernels of long portions that share out rows: token tiles of the causal convolution with a remainder, norms of a warp a group, narrow products of ragged
sizes, and the grouping of more (token, expert) pairs than its threads hold, over several scans of 32 experts."""
import numpy as np
import pytest

from test_gpu_hybrid import F32_TOL, ho, mk, rel, tokens_for  # noqa: F401

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
