"""Logits in pinned memory that a model keeps for its results: arrays that a program holds on to stay as they are, memory comes back and is bounded, also behind a
closed model; prompts in several steps bring the same rows as one."""
import gc

import numpy as np
import pytest

from test_gpu_netusun import F32_TOL, mk, no, rel, tokens_for  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("chunk,tokens", [(16, 90), (64, 65), (256, 90)])
def test_rows_that_are_kept(mk, no, chunk, tokens):  # noqa: F811
    cfg = no.model_config([no.att(), no.lat()], width=40, vocab=5003)
    m, W = mk(cfg, seed=chunk, chunk=chunk)
    toks = [tokens_for(cfg, tokens, k) for k in range(3)]
    exp = [no.run(cfg, W, t)[0] for t in toks]
    got = [m.forward_chunk(t, 0, range(tokens)) for t in toks]      # all three held
    for g, e in zip(got, exp):
        assert rel(g, e) < F32_TOL
    copies, some = [g.copy() for g in got], got[1][3:5]
    del got[1], g
    again = m.forward_chunk(toks[0], 0, range(tokens))
    assert np.array_equal(again, copies[0]) and np.array_equal(got[0], copies[0]) and np.array_equal(got[1], copies[2])
    assert np.array_equal(some, copies[1][3:5])                     # a view keeps its array


def test_memory_is_bounded_and_given_back(mk, no):  # noqa: F811
    cfg = no.model_config([no.att()], width=40, vocab=20011)
    m, _ = mk(cfg, seed=1, chunk=64)
    toks = tokens_for(cfg, 60, 1)
    r = m._results
    whole = list(r.holes)
    held = [m.forward_chunk(toks, 0, range(n)) for n in [20] * 8]    # 1.6 MB each, of 8: the last ones are ordinary arrays
    assert r.live == 6 and sum(h[1] for h in r.holes) < r.MOST and all(np.array_equal(h, held[0]) for h in held)
    del held[1], held[2]
    gc.collect()
    assert r.live == 4
    a, b = m.forward_chunk(toks, 0, range(19)), m.forward_chunk(toks, 0, range(20))
    assert r.live == 6 and np.array_equal(b, held[0]) and np.array_equal(a, b[:19])
    del held, a, b
    gc.collect()
    assert r.live == 1 and r.holes == whole                          # (the decoded token's row)
    rows = m.forward_chunk(toks, 0, range(20))
    want = rows.copy()
    m.close()
    assert np.array_equal(rows, want) and r.base
    del rows
    m._logits = None
    gc.collect()
    assert r.base is None


def test_model_that_is_not_finished(no):  # noqa: F811
    import dsk
    cfg = no.model_config([no.att()], width=40, vocab=97)
    hc, specs = dsk.ARCHITECTURES[cfg["architecture"]](cfg, quant="fp32", max_seq_len=64, chunk=16)
    m = dsk.Model(hc, device=0, layers=specs)
    with pytest.raises(dsk.DskError):
        m.forward_chunk([1, 2, 3], 0, range(3))
    m.close()
