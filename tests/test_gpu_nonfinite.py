"""Infinities and NaN in portions and short steps: what a plain sum over the same numbers gives, and nothing of a token reaches the tokens ahead
of it.  Expected values: the float64 statements, over the tokens ahead where a token's own values are not finite."""
import numpy as np
import pytest

from test_gpu_hybrid import ho  # noqa: F401
from test_gpu_hybrid import mk as mk_hybrid  # noqa: F401
from test_gpu_netusun import F32_TOL, in_portions, mk, no, rel, tokens_for  # noqa: F401
from test_gpu_zetivik import mk as mk_zetivik  # noqa: F401
from test_gpu_zetivik import zo  # noqa: F401

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


# the same where the CTAs of a cluster share a product's depth: the sums of all of them are joined, and looked at, by the CTA that has the row (column: in the first share, one in the
# middle, the ragged last)
@pytest.mark.parametrize("value", [np.inf, np.nan, -3.4e38, 3.39e38])
@pytest.mark.parametrize("tokens,column", [(5, 3), (40, 700), (131, 1099)])
def test_products_of_shared_depth(no, value, tokens, column):  # noqa: F811
    cfg = no.model_config([no.att(heads=2, dim=16, vdim=16, mlp=None)], width=1100, vocab=150)
    W = no.random_weights(cfg, 3)
    toks = tokens_for(cfg, tokens, 3)
    toks[toks == 77] = 5
    exp, layers = no.run(cfg, W, toks)
    h = np.array([no.rms(x, cfg["norm"]["eps"]) * W["final.norm"] for x in layers[-1]])
    W["embed"] = np.array(W["embed"])
    W["embed"][77, column] = value
    with np.errstate(over="ignore", invalid="ignore"):
        col = np.float64(np.float32(value)) * h[:, column] + h @ np.where(np.arange(1100) == column, 0.0, W["embed"][77])
        exp[:, 77] = np.where(np.abs(col) > 3.4028e38, np.copysign(np.inf, col), col) if not np.isnan(value) else np.nan
    m = matrix_model(no, cfg, W, 256)
    got = m.forward_chunk(toks, 0, range(tokens))
    m.close()
    others = np.arange(150) != 77
    assert rel(got[:, others], exp[:, others]) < F32_TOL
    fin = np.isfinite(exp[:, 77])
    near = np.abs(np.abs(col) / 3.4028e38 - 1.0) < 1e-3 if np.isfinite(value) else np.zeros(tokens, bool)
    assert np.array_equal(got[~fin & ~near, 77], exp[~fin & ~near, 77], equal_nan=True)
    if np.any(fin & ~near):
        assert np.all(np.abs(got[fin & ~near, 77] - exp[fin & ~near, 77]) <= 1e-4 * np.abs(value))


def poisoned(W, value, row):
    W["embed"][row, 1] = value


def ahead_of_the_poison(m, run, cfg, W, toks, at, sizes):
    """Largest error of the tokens ahead of token `at` (the head is the embedding: the poisoned row's own logits are left out)."""
    others = np.arange(cfg["vocab"]) != toks[at]
    with np.errstate(invalid="ignore"):
        got, exp = in_portions(m, toks, sizes)[:at, others], run(cfg, W, toks[:at])[0][:, others]
    return rel(got, exp) if np.all(np.isfinite(got)) else np.inf


def attention_model(mk, no, kind, value):  # noqa: F811
    layer = {"grouped": lambda: no.att(heads=6, kv_heads=2, dim=12, vdim=10, size=25), "own_keys": lambda: no.att(heads=3, kv_heads=3, dim=16, vdim=70, size=None, conv=1),
             "latent": lambda: no.lat(heads=3), "deep_latent": lambda: no.lat(heads=9, kv_rank=300, rot_dim=6)}[kind]
    cfg = no.model_config([layer(), layer()], width=48, vocab=97)
    return (cfg,) + mk(cfg, seed=4, chunk=64, edit=lambda W: poisoned(W, value, 90))


def check_steps(mk, no, kind, value, steps):  # noqa: F811
    """A step whose token `at` has keys and values that are not finite: its earlier tokens share CTAs and key tiles with it."""
    cfg, m, W = attention_model(mk, no, kind, value)
    for sizes in steps:
        n = sum(sizes)
        toks = tokens_for(cfg, n, 5)
        toks[toks == 90] = 7
        for at in (1, 6, 15, n - 1):
            t = toks.copy()
            t[at] = 90
            m.reset()
            assert ahead_of_the_poison(m, no.run, cfg, W, t, at, sizes) < F32_TOL


@pytest.mark.parametrize("value", [np.inf, np.nan])
@pytest.mark.parametrize("kind", ["grouped", "own_keys", "latent", "deep_latent"])
def test_attention_of_portions(mk, no, kind, value):  # noqa: F811
    check_steps(mk, no, kind, value, [[40], [64], [33, 32]])


@pytest.mark.parametrize("value", [np.inf, np.nan])
@pytest.mark.parametrize("kind", ["grouped", "own_keys", "latent", "deep_latent"])
def test_attention_of_short_steps(mk, no, kind, value):  # noqa: F811
    check_steps(mk, no, kind, value, [[2] * 20, [3] * 13, [5] * 8, [8] * 5, [13] * 3, [31, 9]])


@pytest.mark.parametrize("value", [np.inf, np.nan])
def test_latents_in_bf16(mk_hybrid, ho, value):  # noqa: F811
    """Latent attention of bf16 models (one bf16 part an operand) against the same portion without the token."""
    att = {"type": "latent_attention", "mixer": {"heads": 3, "dim": 12, "vdim": 20, "kv_rank": 40, "mask": {"size": 30}, "scale": 0.3}, "mlp": None}
    cfg = ho.small_config(layers=[att] * 2, width=36, norm={"eps": 1e-5, "groups": 1})
    m, W = mk_hybrid(cfg, seed=4, quant="bf16", chunk=64, edit=lambda W: poisoned(W, value, 50))
    toks = tokens_for(cfg, 64, 5)
    toks[toks == 50] = 7
    base = m.forward_chunk(toks, 0, range(64))
    for at in (1, 16, 33, 63):
        t = toks.copy()
        t[at] = 50
        m.reset()
        got = m.forward_chunk(t, 0, range(64))
        others = np.arange(cfg["vocab"]) != 50
        assert np.all(np.isfinite(got[:at, others])) and rel(got[:at, others], base[:at, others]) < 2e-2   # (rows that are summed again: weights not rounded)
    m.reset()


# heads of 64 entries and more (pattn5): blocks of 64 and 128 value columns, depth in one, two and three pieces, one block of queries and several, whose rows in front of the token share
# a tile with it
@pytest.mark.parametrize("value", [np.inf, np.nan])
@pytest.mark.parametrize("kind", ["grouped", "own_keys", "latent", "deep_latent"])
def test_attention_of_wide_heads(mk, no, kind, value):  # noqa: F811
    layer = {"grouped": lambda: no.att(heads=4, kv_heads=2, dim=64, vdim=64, size=50), "own_keys": lambda: no.att(heads=2, kv_heads=2, dim=100, vdim=150, size=None),
             "latent": lambda: no.lat(heads=2, dim=64, rot_dim=8, vdim=70), "deep_latent": lambda: no.lat(heads=2, dim=128, rot_dim=64, vdim=128)}[kind]
    cfg = no.model_config([layer(), layer()], width=48, vocab=97)
    m, W = mk(cfg, seed=4, chunk=256, edit=lambda W: poisoned(W, value, 90))
    for sizes in ([40], [200], [70, 90]):
        n = sum(sizes)
        toks = tokens_for(cfg, n, 5)
        toks[toks == 90] = 7
        for at in (1, 31, n // 2 + 3, n - 1):
            t = toks.copy()
            t[at] = 90
            m.reset()
            assert ahead_of_the_poison(m, no.run, cfg, W, t, at, sizes) < F32_TOL
    m.reset()


@pytest.mark.parametrize("value", [np.inf, np.nan])
@pytest.mark.parametrize("kind", ["grouped", "own_keys", "latent"])
def test_shares_of_the_keys_of_wide_heads(mk, no, kind, value):  # noqa: F811
    layer = {"grouped": lambda: no.att(heads=4, kv_heads=2, dim=64, vdim=64, size=None), "own_keys": lambda: no.att(heads=2, kv_heads=2, dim=100, vdim=150, size=300),
             "latent": lambda: no.lat(heads=2, dim=64, rot_dim=8, vdim=128)}[kind]
    cfg = no.model_config([layer(), layer()], width=48, vocab=97)
    m, W = mk(cfg, seed=4, chunk=300, context=700, edit=lambda W: poisoned(W, value, 90))
    toks = tokens_for(cfg, 560, 5)
    toks[toks == 90] = 7
    for at in (20, 420, 500, 558):
        t = toks.copy()
        t[at] = 90
        m.reset()
        assert ahead_of_the_poison(m, no.run, cfg, W, t, at, [300, 100, 160]) < F32_TOL
    m.reset()


@pytest.mark.parametrize("value", [np.inf, np.nan])
@pytest.mark.parametrize("dim,vdim,size,sizes", [(64, 64, 30, [130]), (128, 128, 400, [300, 40])])   # (300 keys behind 40 queries: shares)
def test_latents_of_wide_heads_in_bf16(mk_hybrid, ho, value, dim, vdim, size, sizes):  # noqa: F811
    att = {"type": "latent_attention", "mixer": {"heads": 3, "dim": dim, "vdim": vdim, "kv_rank": 40, "mask": {"size": size}, "scale": 0.1}, "mlp": None}
    cfg = ho.small_config(layers=[att] * 2, width=36, norm={"eps": 1e-5, "groups": 1})
    m, W = mk_hybrid(cfg, seed=4, quant="bf16", chunk=300, context=500, edit=lambda W: poisoned(W, value, 50))
    n = sum(sizes)
    toks = tokens_for(cfg, n, 5)
    toks[toks == 50] = 7
    base = in_portions(m, toks, sizes)
    for at in (1, 33, n // 2, n - 1):
        t = toks.copy()
        t[at] = 50
        m.reset()
        got = in_portions(m, t, sizes)
        others = np.arange(cfg["vocab"]) != 50
        assert np.all(np.isfinite(got[:at, others])) and rel(got[:at, others], base[:at, others]) < 2e-2   # (rows that are summed again: weights not rounded)
    m.reset()


@pytest.mark.parametrize("value", [np.inf, np.nan])
def test_recurrence_in_blocks(mk_hybrid, ho, value):  # noqa: F811
    ssd = {"type": "mamba2", "mixer": {"heads": 4, "vdim": 12, "state": 33, "groups": 2, "conv": 3, "norm_groups": 1}, "mlp": None}
    cfg = ho.small_config(layers=[ssd] * 2, width=36, norm={"eps": 1e-5, "groups": 1})
    m, W = mk_hybrid(cfg, seed=4, chunk=64, edit=lambda W: poisoned(W, value, 50))
    toks = tokens_for(cfg, 40, 5)
    toks[toks == 50] = 7
    for sizes in ([40], [17, 23], [5] * 8):
        for at in (1, 9, 20, 39):
            t = toks.copy()
            t[at] = 50
            m.reset()
            assert ahead_of_the_poison(m, ho.run, cfg, W, t, at, sizes) < F32_TOL
    m.reset()


@pytest.mark.parametrize("value", [np.inf, np.nan])
def test_recurrence_in_segments(mk_hybrid, ho, value):  # noqa: F811
    ssd = {"type": "mamba2", "mixer": {"heads": 3, "vdim": 20, "state": 64, "groups": 1, "conv": 3, "norm_groups": 1}, "mlp": None}
    cfg = ho.small_config(layers=[ssd] * 2, width=36, norm={"eps": 1e-5, "groups": 1})
    m, W = mk_hybrid(cfg, seed=4, chunk=400, edit=lambda W: poisoned(W, value, 50))
    toks = tokens_for(cfg, 400, 5)
    toks[toks == 50] = 7
    for at in (1, 30, 201, 399):
        t = toks.copy()
        t[at] = 50
        m.reset()
        assert ahead_of_the_poison(m, ho.run, cfg, W, t, at, [400]) < F32_TOL
    m.reset()


def segments_model(kind, mk, no, mk_zetivik, zo, edit):  # noqa: F811
    """Recurrences whose walks run in segments on the tensor cores: (oracle's run, config, model, weights)."""
    if kind.startswith("lightning"):
        heads, dim, vdim = (3, 64, 20) if kind == "lightning_64" else (2, 128, 68)
        cfg = zo.model_config([zo.light(heads=heads, dim=dim, vdim=vdim, decay=[0.999, 1.0, 0.5][:heads])], width=40, vocab=97)
        return (zo.run, cfg) + mk_zetivik(cfg, seed=4, chunk=500, edit=edit)
    heads, dim, vdim = (3, 64, 64) if kind == "matrix_64" else (2, 128, 12)
    cfg = no.model_config([no.mem(heads=heads, dim=dim, vdim=vdim)], width=40, vocab=97)
    return (no.run, cfg) + mk(cfg, seed=4, chunk=500, edit=edit)


@pytest.mark.parametrize("value", [np.inf, np.nan])
@pytest.mark.parametrize("kind", ["lightning_64", "lightning_128", "matrix_64", "matrix_128"])
def test_walks_in_segments(mk, no, mk_zetivik, zo, kind, value):  # noqa: F811
    run, cfg, m, W = segments_model(kind, mk, no, mk_zetivik, zo, lambda W: poisoned(W, value, 50))
    toks = tokens_for(cfg, 500, 5)
    toks[toks == 50] = 7
    for at in (1, 66, 200, 499):
        t = toks.copy()
        t[at] = 50
        m.reset()
        assert ahead_of_the_poison(m, run, cfg, W, t, at, [500]) < F32_TOL
    m.reset()


@pytest.mark.parametrize("kind", ["lightning_64", "lightning_128", "matrix_64", "matrix_128"])
def test_values_past_bfloat16_in_segments(mk, no, mk_zetivik, zo, kind):  # noqa: F811
    """One value of one token next to the largest fp32 number, finite but an infinity in bfloat16, against keys and queries so small that what it leaves in the state
    is ordinary: blocks with such a value update the state by fused multiply-adds, the first one of a segment too."""
    largest = 3.3985e38                                      # (bfloat16 rounds to an infinity from 3.3962e38 on)

    def edit(W):
        W["embed"] = np.array(W["embed"])
        W["embed"][:, 3] = W["embed"][:, 5] = 0.0            # columns that token 50 has to itself: the value's weights read nothing else
        W["embed"][50, 3], W["embed"][50, 5] = 3.0, 0.125
        h = zo.rms(W["embed"][50], cfg_eps) * (1.0 + W["l0.norm1"] if kind.startswith("lightning") else W["l0.norm1"])
        for n in "qk":
            W["l0.mix." + n] = W["l0.mix." + n] * 1e-18
        v = np.array(W["l0.mix.v"])
        v[2] = 0.0
        v[2, 3] = zo.bf16_to_f64(zo.to_bf16(np.array([0.995 * largest / h[3]])))[0]
        v[2, 5] = (largest - v[2, 3] * h[3]) / h[5]
        W["l0.mix.v"] = v
        if kind.startswith("matrix"):
            W["l0.mix.f.b"] = W["l0.mix.f.b"] * 0.0 + 8.0    # (kept for the rest of the sequence)
    cfg_eps = 1e-5
    run, cfg, m, W = segments_model(kind, mk, no, mk_zetivik, zo, edit)
    assert cfg["norm"]["eps"] == cfg_eps
    toks = tokens_for(cfg, 500, 5)
    toks[toks == 50] = 7
    for at in (2, 64, 130, 260, 450):
        t = toks.copy()
        t[at] = 50
        exp = run(cfg, W, t)[0]
        assert np.all(np.isfinite(exp))
        m.reset()
        assert rel(in_portions(m, t, [500]), exp) < F32_TOL
    m.reset()


@pytest.mark.parametrize("router", ["sigmoid", "groups"])
def test_routed_rows(mk, mk_hybrid, no, ho, router):  # noqa: F811
    """A token whose router scores are NaN gets experts that exist, and the others theirs: in short steps, and in portions, where rows are put into
    expert order."""
    if router == "groups":
        cfg, run = no.model_config([no.att(mlp=no.moe(experts=12, top=4, count=3, keep=2))], width=40, vocab=97), no.run
        m, W = mk(cfg, seed=4, chunk=64, edit=lambda W: poisoned(W, np.nan, 50))
    else:
        moe = {"kind": "moe", "router": {"experts": 7, "top": 3, "scale": 1.0}, "expert": {"ff": 12, "limit": 3.0}}
        att = {"type": "latent_attention", "mixer": {"heads": 3, "dim": 12, "vdim": 20, "kv_rank": 40, "mask": {"size": 30}, "scale": 0.3}, "mlp": moe}
        cfg, run = ho.small_config(layers=[att], width=36, norm={"eps": 1e-5, "groups": 1}), ho.run
        m, W = mk_hybrid(cfg, seed=4, chunk=64, edit=lambda W: poisoned(W, np.nan, 50))
    toks = tokens_for(cfg, 60, 5)
    toks[toks == 50] = 7
    for sizes in ([60], [4] * 15, [9, 51]):
        for at in (1, 20, 59):
            t = toks.copy()
            t[at] = 50
            m.reset()
            assert ahead_of_the_poison(m, run, cfg, W, t, at, sizes) < F32_TOL


@pytest.mark.parametrize("value", [np.inf, np.nan])
@pytest.mark.parametrize("kind", ["grouped", "own_keys", "deep_latent"])
def test_shares_of_the_keys(mk, no, kind, value):  # noqa: F811
    """The same where a portion's keys are cut into shares: rows ahead of the token take part in its share too."""
    layer = {"grouped": lambda: no.att(heads=4, kv_heads=2, dim=12, vdim=10, size=None), "own_keys": lambda: no.att(heads=2, kv_heads=2, dim=16, vdim=70, size=200, conv=1),
             "deep_latent": lambda: no.lat(heads=2, kv_rank=30, rot_dim=6)}[kind]
    cfg = no.model_config([layer(), layer()], width=48, vocab=97)
    m, W = mk(cfg, seed=4, chunk=300, context=700, edit=lambda W: poisoned(W, value, 90))
    toks = tokens_for(cfg, 560, 5)
    toks[toks == 90] = 7
    for at in (420, 500, 558):
        t = toks.copy()
        t[at] = 90
        m.reset()
        assert ahead_of_the_poison(m, no.run, cfg, W, t, at, [300, 100, 160]) < F32_TOL
