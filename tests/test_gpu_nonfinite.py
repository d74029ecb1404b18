"""Infinities and NaN in portions and short steps: what a plain sum over the same numbers gives, and nothing of a token reaches the tokens ahead
of it.  Expected values: the float64 statements, over the tokens ahead where a token's own values are not finite."""
import numpy as np
import pytest

from test_gpu_netusun import F32_TOL, no, rel, tokens_for  # noqa: F401

pytestmark = pytest.mark.gpu


def matrix_model(no, cfg, W, chunk):  # noqa: F811
    """A model with fp32 matrices (a checkpoint's are bfloat16)."""
    import dsk
    hc, specs = dsk.ARCHITECTURES[cfg["architecture"]](cfg, quant="fp32", max_seq_len=256, chunk=chunk)
    m = dsk.Model(hc, device=0, layers=specs)
    for name, w in W.items():
        a = np.asarray(w, np.float32)
        m.upload(name, "F32", a.shape, a)
    m.finalize()
    return m


# value: one weight of a row of the head.  3.4e38 is past the largest bfloat16 number, a finite fp32 one
@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan, 3.4e38, -3.4e38, 3.39e38])
@pytest.mark.parametrize("tokens", [5, 64, 131])
def test_products(no, value, tokens):  # noqa: F811
    cfg = no.model_config([no.att(heads=2, dim=16, vdim=16, mlp=no.dense(112))], width=100, vocab=150)
    W = no.random_weights(cfg, 3)
    toks = tokens_for(cfg, tokens, 3)
    toks[toks == 77] = 5                                     # (the head is the embedding: row 77 is read by the head alone)
    exp = no.run(cfg, W, toks)[0]
    h = np.linalg.lstsq(np.asarray(W["embed"]), exp.T, rcond=None)[0].T          # the rows that the head multiplies
    W["embed"] = np.array(W["embed"])
    W["embed"][77, 40] = value
    with np.errstate(over="ignore", invalid="ignore"):
        col = np.float64(np.float32(value)) * h[:, 40] + h @ np.where(np.arange(100) == 40, 0.0, W["embed"][77])
        exp[:, 77] = np.where(np.abs(col) > 3.4028e38, np.copysign(np.inf, col), col) if not np.isnan(value) else np.nan
    m = matrix_model(no, cfg, W, 256)
    got = m.forward_chunk(toks, 0, range(tokens))
    m.close()
    others = np.arange(150) != 77
    assert rel(got[:, others], exp[:, others]) < F32_TOL
    fin = np.isfinite(exp[:, 77])
    near = np.abs(np.abs(col) / 3.4028e38 - 1.0) < 1e-3 if np.isfinite(value) else np.zeros(tokens, bool)   # (either side of the overflow)
    assert np.array_equal(got[~fin & ~near, 77], exp[~fin & ~near, 77], equal_nan=True)
    if np.any(fin & ~near):
        assert np.all(np.abs(got[fin & ~near, 77] - exp[fin & ~near, 77]) <= 1e-4 * np.abs(value))
