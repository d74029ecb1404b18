"""Logits on their way to the host, bit for bit: through the state's two pinned pieces of 256 KB (pageable memory: one piece, two, many with a ragged end
behind them), straight into pinned memory, and row by row."""
import ctypes as C

import numpy as np
import pytest
import torch

from test_gpu_netusun import mk, no, tokens_for  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("vocab,tokens", [(4097, 16), (4099, 31), (3001, 200), (9973, 300)])   # 256 KB and 256 bytes, two pieces, 9.2, 39 in groups of 256 rows
def test_destinations(mk, no, vocab, tokens):  # noqa: F811
    import dsk
    cfg = no.model_config([no.att()], width=40, vocab=vocab)
    m, _ = mk(cfg, seed=vocab, chunk=512)
    toks = tokens_for(cfg, tokens, 3)
    want = np.arange(tokens, dtype=np.int32)

    def into(ptr):
        m.reset()
        return m.L.dsk_forward_chunk(m.h, m.s, toks.ctypes.data_as(dsk.i32p), tokens, 0, want.ctypes.data_as(dsk.i32p), tokens, C.cast(ptr, dsk.f32p), None)

    got = m.forward_chunk(toks, 0, range(tokens))
    pinned = torch.zeros(tokens, vocab, pin_memory=True)
    assert into(pinned.data_ptr()) == 0 and np.array_equal(pinned.numpy(), got)
    dev = torch.zeros(tokens, vocab, device="cuda:0")           # not a host address: an error of the call, or the rows
    torch.cuda.synchronize()
    if into(dev.data_ptr()) == 0:
        assert np.array_equal(dev.cpu().numpy(), got)
    m.reset()
    some = m.forward_chunk(toks, 0, [0, tokens // 2, tokens - 1])
    assert np.abs(some - got[[0, tokens // 2, tokens - 1]]).max() < 1e-5 * np.abs(got).max()   # (a product of three rows sums in another order)
